"""A refinement step of three folded iterations keeps its directions instead
of the correction: the bits of the separate updates, in the row form and the
flat form of the update, and of other iteration counts' steps before and
after it."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n_b", [((12, 20, 210), 1), ((18, 33, 197), 5), ((40, 31, 33), 2)])
def test_same_bits(shape, n_b):
    from ion_gym_gb300.physics.mixed import MixedSession
    rng = np.random.default_rng(shape[0])
    masks = []
    for _ in range(n_b):
        m = np.zeros(shape, bool)
        lo = [int(rng.integers(1, max(2, s - s // 3))) for s in shape]
        m[tuple(slice(a, a + max(2, s // 5)) for a, s in zip(lo, shape))] = True
        masks.append(m)
    box = np.zeros(shape, bool)
    box[0] = box[-1] = True
    metal = np.any(masks, 0) | box
    got = {}
    for fold in ("0", "1"):
        os.environ["IG_MIXED_FOLD"] = fold
        try:
            with MixedSession(metal, n_b) as s:
                got[fold] = []
                for iters in (3, 5, 3, 2):
                    s.set_cycle(2, 2, iters)
                    got[fold].append(s.solve_bases(masks, 1.0, 1e-9).copy())
        finally:
            del os.environ["IG_MIXED_FOLD"]
    for a, b in zip(got["0"], got["1"]):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
