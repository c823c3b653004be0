"""A problem's bits do not depend on the batch it is solved in: the partial sums
of the flexible CG follow the grid alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# grids of fewer, some and many more groups of slots than the least blocks'
# threads take; a flat one (its dot products by k_cg_dot); problems of one deck,
# so that a batch takes the steps that one takes
@pytest.mark.parametrize("shape", [(12, 20, 210), (33, 41, 27), (64, 80, 72), (129, 97, 90),
                                   (1, 150, 170)])
def test_alone_and_in_batches(shape):
    from ion_gym_gb300.physics.mixed import MixedSession
    rng = np.random.default_rng(shape[2])
    mask = np.zeros(shape, bool)
    for _ in range(3):
        lo = [int(rng.integers(0, max(1, s - s // 4))) for s in shape]
        mask[tuple(slice(a, a + max(1, s // 6)) for a, s in zip(lo, shape))] = True
    metal = mask.copy()
    metal[..., 0] = metal[..., -1] = True
    mask[..., 0] = mask[..., -1] = False
    vals = np.where(mask, rng.uniform(-1.0, 1.0, shape), 0.0)
    with MixedSession(metal, 24) as s:
        s.set_cycle(2, 2, 3)
        basis = s.solve_bases([mask], 1.0, 1e-9)[0].copy()
        field = s.solve_values(vals[None], 1e-9)[0].copy()
        for n in (2, 7, 24):
            got = s.solve_bases([mask] * n, 1.0, 1e-9)
            assert all(np.array_equal(g.view(np.uint64), basis.view(np.uint64)) for g in got)
            got = s.solve_values(np.stack([vals] * n), 1e-9)
            assert all(np.array_equal(g.view(np.uint64), field.view(np.uint64)) for g in got)
