"""The masks of every level from one launch a level: decks with one-node
plates at odd and even positions on even, odd and short axes solve to the
FP64 V-cycle's potentials, and after a rebind to the bits of a new session."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACC = 1e-9


def _deck(shape, seed):
    rng = np.random.default_rng(seed)
    fixed = np.zeros(shape, bool)
    val = np.zeros(shape)
    for a in range(3):
        if shape[a] > 2:
            fixed[(slice(None),) * a + (0,)] = fixed[(slice(None),) * a + (-1,)] = True
    for q in range(4):                      # one-node plates across z, ragged extents
        k = int(rng.integers(1, shape[2] - 1))
        i0, j0 = int(rng.integers(0, shape[0] // 2)), int(rng.integers(0, shape[1] // 2))
        plate = (slice(i0, i0 + max(1, shape[0] // 2)), slice(j0, j0 + max(1, shape[1] // 2)), k)
        fixed[plate] = True
        val[plate] = float(rng.uniform(-1, 1))
    return fixed, val


@pytest.mark.parametrize("shape", [(33, 34, 51), (20, 47, 90), (2, 40, 65)])
def test_plates(shape):
    from ion_gym_gb300.physics import multigrid3d as M
    from ion_gym_gb300.physics.mixed import MixedSession
    decks = [_deck(shape, s) for s in range(4)]
    f = [np.stack([decks[a][0], decks[b][0]]) for a, b in ((0, 1), (2, 3))]
    v = [np.stack([decks[a][1], decks[b][1]]) for a, b in ((0, 1), (2, 3))]
    span = np.array([2.0, 2.0])
    with MixedSession(f[0]) as s:
        first = s.solve_values(v[0], ACC, span=span).copy()
        s.rebind(f[1])
        again = s.solve_values(v[1], ACC, span=span).copy()
    with MixedSession(f[1]) as s:
        fresh = s.solve_values(v[1], ACC, span=span)
        assert np.array_equal(again.view(np.uint64), fresh.view(np.uint64))
    for q in range(2):
        ref = M.solve3d_vmg(decks[q][0], decks[q][1], tol=2e-13, max_cycles=400,
                            accept_stagnation=True)[0]
        assert np.abs(first[q] - ref).max() <= ACC * span[q]
