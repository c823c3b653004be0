"""The basis door's device-side set-up: flip symmetries found on the device
(plain, per axis, broken by one node of the mask or of the metal, axes too
short to count), bases whose values are given by a mask alone, a voltage that
is 0 or NaN, and worker threads that come and go."""
import threading

import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _symmetric(shape):
    fixed = np.zeros(shape, bool)
    fixed[0] = fixed[-1] = True
    fixed[:, 0] = fixed[:, -1] = True
    core = tuple(slice(n // 3, n - n // 3) for n in shape)
    val = np.zeros(shape)
    fixed[core] = True
    val[core] = 1e4
    return fixed, val


@pytest.mark.parametrize("shape", [(33, 34, 21), (20, 2, 19), (17, 18, 1)])
def test_symmetries(shape):
    from ion_gym_gb300.physics import multigrid3d as M
    fixed, val = _symmetric(shape)
    decks = [(fixed, val)]
    f, v = fixed.copy(), val.copy()
    p = tuple(min(1, n - 1) for n in shape)
    f[p] = True                                     # the metal breaks it
    decks.append((f, v))
    v = val.copy()
    v[0, shape[1] // 4, 0] = 5.0                    # a value breaks it
    decks.append((fixed, v))
    for f, v in decks:
        a = M.solve3d_vmg(f, v, tol=1e-5, accept_stagnation=True)
        b = port.solve3d_vmg(f, v, tol=1e-5, accept_stagnation=True)
        assert a[1:] == b[1:] and same_bits(a[0], b[0])


def test_bases_by_mask():
    from ion_gym_gb300.physics import multigrid3d as M, solver3d as S
    fixed, val = _symmetric((21, 20, 23))
    masks = {1: val > 0, 2: fixed & ~(val > 0)}
    for v in (1e4, -3.0):
        a, b = (m.solve_bases_mg(masks, v_basis=v, tol=1e-4) for m in (M, port))
        assert all(same_bits(a[i], b[i]) for i in masks)
        a = S.solve_bases(masks, v_basis=v, tol=1e-2)
        b = port.solve_bases(masks, v_basis=v, tol=1e-2)
        assert all(same_bits(a[i], b[i]) for i in masks)
    zero = M.solve_bases_mg(masks, v_basis=0.0, tol=1e-4)
    assert not zero[1].any() and not zero[2].any()


def test_threads_come_and_go():
    """Solves from 24 short-lived threads, a few at a time."""
    from ion_gym_gb300.physics import multigrid3d as M
    fixed, val = _symmetric((19, 21, 20))
    want = port.solve3d_vmg(fixed, val, tol=1e-5)[0]
    got = []

    def work():
        got.append(M.solve3d_vmg(fixed, val, tol=1e-5)[0])

    for _ in range(6):
        ts = [threading.Thread(target=work) for _ in range(4)]
        [t.start() for t in ts]
        [t.join() for t in ts]
    assert len(got) == 24 and all(same_bits(g, want) for g in got)
