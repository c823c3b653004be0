"""solve3d's loop as one resident launch (grids of up to 1.2 million slots a
colour) and above it as launched sweeps: phi, pairs and the last delta equal
the oracle's, at one node a thread and several, on flat axes, at the sweep
cap, from a given start, and when solves run from several threads at once."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _deck(shape, seed):
    rng = np.random.default_rng(seed)
    fixed = rng.random(shape) < 0.01
    fixed[0] = True
    fixed[tuple(n // 2 for n in shape)] = True
    return fixed, np.where(fixed, rng.uniform(-100, 100, shape), 0.0)


# 160 x 128 x 125 has 1.29 million slots (launched); 140 x 128 x 125 1.13
@pytest.mark.parametrize("shape", [(5, 4, 3), (1, 40, 33), (33, 1, 1), (70, 64, 65),
                                   (140, 128, 125), (160, 128, 125)])
def test_solve3d(shape):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck(shape, 11)
    a = S.solve3d(fixed, val, tol=1e-3, omega=1.5)
    b = port.solve3d(fixed, val, tol=1e-3, omega=1.5)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])


def test_start_cap_and_nan():
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck((41, 40, 39), 12)
    start = np.random.default_rng(1).uniform(-10, 10, fixed.shape)
    a = S.solve3d(fixed, val, tol=1e-4, omega=1.7, phi0=start)
    b = port.solve3d(fixed, val, tol=1e-4, omega=1.7, phi0=start)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])
    with pytest.raises(S.SolveNotConverged, match="cap of 5 sweeps"):
        S.solve3d(fixed, val, tol=1e-12, max_sweeps=5)
    # the reference's maximum never takes a NaN: such a solve stops on the rest
    val = val.copy()
    val[0, 0, 0] = np.nan
    a = S.solve3d(fixed, val, tol=1e-4, omega=1.5)
    b = port.solve3d(fixed, val, tol=1e-4, omega=1.5)
    assert a[1:] == b[1:] and np.array_equal(np.isnan(a[0]), np.isnan(b[0]))


def test_solves_from_several_threads():
    from ion_gym_gb300.physics import solver3d as S
    decks = [_deck((40 + 3 * q, 37, 44), q) for q in range(6)]
    with ThreadPoolExecutor(6) as ex:
        got = list(ex.map(lambda d: S.solve3d(*d, tol=1e-3, omega=1.5), decks))
    for (f, v), a in zip(decks, got):
        b = port.solve3d(f, v, tol=1e-3, omega=1.5)
        assert a[1:] == b[1:] and same_bits(a[0], b[0])


# shared memory from a few KB to over 100 a CTA, in calls of threads that
# start theirs at any time
def test_threads_with_small_and_large_grids():
    from ion_gym_gb300.physics import solver3d as S
    decks = [_deck(shape, 30 + q) for q, shape in enumerate([(40, 40, 40), (129, 129, 129)] * 3)]
    want = [S.solve3d(*d, tol=0.5, omega=1.5) for d in decks]

    def calls(q):
        for _ in range(40 if q % 2 == 0 else 15):
            a = S.solve3d(*decks[q], tol=0.5, omega=1.5)
            assert a[1:] == want[q][1:] and same_bits(a[0], want[q][0])

    with ThreadPoolExecutor(len(decks)) as ex:
        list(ex.map(calls, range(len(decks))))


def test_solves_beside_a_session():
    """The loop makes room for a session's kernels between its turns and takes
    up again where the launched sweeps left: the same bits as alone."""
    from ion_gym_gb300.physics import solver3d as S
    from ion_gym_gb300.physics.mixed import MixedSession
    decks = [_deck(shape, 50 + q) for q, shape in enumerate([(65, 64, 63), (97, 96, 95)])]
    want = [S.solve3d(*d, tol=1e-6, omega=1.8) for d in decks]
    fixed, val = _deck((64, 64, 64), 60)
    with MixedSession(fixed, 1) as s:
        field = s.solve_values(val[None], 1e-9)

        def sessions(_):
            for _ in range(20):
                assert same_bits(s.solve_values(val[None], 1e-9), field)

        def solves(q):
            for _ in range(6):
                a = S.solve3d(*decks[q], tol=1e-6, omega=1.8)
                assert a[1:] == want[q][1:] and same_bits(a[0], want[q][0])

        with ThreadPoolExecutor(3) as ex:
            jobs = [ex.submit(sessions, 0)] + [ex.submit(solves, q) for q in (0, 1)]
            for j in jobs:
                j.result()
    for (f, v), a in zip(decks, want):
        b = port.solve3d(f, v, tol=1e-6, omega=1.8)
        assert a[1:] == b[1:] and same_bits(a[0], b[0])
