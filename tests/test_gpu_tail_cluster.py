"""The small levels of a mixed cycle in one cluster launch per problem
(k_tail_cluster) against the separate launches."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

V, ACC = 1.0, 1e-9


def _deck(shape, seed, n):
    rng = np.random.default_rng(seed)
    masks = []
    for _ in range(n):
        m = np.zeros(shape, bool)
        lo = [int(rng.integers(0, max(1, s - max(2, s // 4)))) for s in shape]
        m[tuple(slice(a, a + max(2, s // 5)) for a, s in zip(lo, shape))] = True
        masks.append(m)
    return masks


# levels of 32 x 40 x 36 nodes (one group of slots for most threads), 45^3
# (past the cluster's share: it starts a level further down), a short axis,
# odd and even extents, one CTA's worth (12^3 above the bottom), one problem
@pytest.mark.parametrize("shape,n_b,cycle", [
    (shape, n_b, cycle)
    for shape, n_b in [((64, 80, 72), 3), ((90, 90, 90), 2), ((9, 121, 90), 3), ((33, 41, 27), 1)]
    for cycle in [(2, 2, 3), (1, 2, 3), (3, 2, 2)]] + [((47, 46, 48), 9, (2, 2, 3))])
def test_cluster_gives_the_separate_launches_bits(shape, n_b, cycle):
    from ion_gym_gb300.physics.mixed import MixedSession
    masks = _deck(shape, 11, n_b)
    metal = np.zeros(shape, bool)
    for m in masks:
        metal |= m
    got = {}
    for tail in ("0", "1"):
        os.environ["IG_MIXED_TAIL"] = tail
        try:
            with MixedSession(metal, n_b) as s:
                s.set_cycle(*cycle)
                got[tail] = s.solve_bases(masks, V, ACC)
        finally:
            del os.environ["IG_MIXED_TAIL"]
    assert np.array_equal(got["0"].view(np.uint64), got["1"].view(np.uint64))
