"""Solves with surface fractions whose cut nodes are few take the listed
form (the plain update plus a list of cut nodes): the same bits as the
oracle for every shape, stencil and driver, at both sides of the rule (no
cut node, a few, just under and over a tenth of the grid) and where halving
a value would round (subnormal potentials)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _deck(shape, cut, seed, v=100.0):
    """A block in a box grounded on its low-x face, other faces reflecting;
    `cut` of the free nodes have one short leg or more."""
    rng = np.random.default_rng(seed)
    fixed = np.zeros(shape, bool)
    fixed[0] = True
    core = tuple(slice(n // 3, max(n // 3 + 1, n // 2)) for n in shape)
    fixed[core] = True
    val = np.zeros(shape)
    val[core] = v
    th = np.ones((6,) + shape, np.float32)
    free = np.flatnonzero(~fixed.ravel())
    pick = rng.choice(free, int(round(cut * free.size)), replace=False)
    flat = th.reshape(6, -1)
    for p in pick:
        legs = rng.integers(0, 6, rng.integers(1, 4))
        flat[legs, p] = rng.uniform(1e-3, 0.999, legs.size).astype(np.float32)
    return fixed, val, th


@pytest.mark.parametrize("stencil", ["ghost_linear", "sw"])
@pytest.mark.parametrize("shape,cut", [((33, 21, 18), 0.0), ((33, 21, 18), 0.01),
                                       ((19, 34, 27), 0.09), ((19, 34, 27), 0.2),
                                       ((17, 16, 1), 0.05), ((9, 2, 40), 0.03)])
def test_solve3d_with_few_cut_nodes(shape, cut, stencil):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val, th = _deck(shape, cut, 3)
    # omega 1: Gauss-Seidel converges whatever the legs
    a = S.solve3d(fixed, val, theta=th, tol=1e-6, stencil=stencil, omega=1.0)
    b = port.solve3d(fixed, val, theta=th, tol=1e-6, stencil=stencil, omega=1.0)
    assert np.isfinite(b[0]).all()
    assert a[1:] == b[1:] and same_bits(a[0], b[0])


@pytest.mark.parametrize("stencil", ["ghost_linear", "sw"])
def test_vcycle_and_cascadic_with_few_cut_nodes(stencil):
    from ion_gym_gb300.physics import multigrid3d as M
    fixed, val, th = _deck((33, 34, 29), 0.002, 5)
    a = M.solve3d_vmg(fixed, val, theta=th, tol=1e-5, stencil=stencil)
    b = port.solve3d_vmg(fixed, val, theta=th, tol=1e-5, stencil=stencil)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])
    for levels in (1, 3):
        a = M.solve3d_mg(fixed, val, theta=th, tol=1e-6, stencil=stencil, max_levels=levels)
        b = port.solve3d_mg(fixed, val, theta=th, tol=1e-6, stencil=stencil, max_levels=levels)
        assert a[1:] == b[1:] and same_bits(a[0], b[0])


@pytest.mark.parametrize("v", [3e-322, 7e-308, 1e-290])
def test_subnormal_potentials(v):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val, th = _deck((15, 14, 13), 0.03, 7, v)
    a = S.solve3d(fixed, val, theta=th, tol=v * 0.02, stencil="sw", omega=1.0)
    b = port.solve3d(fixed, val, theta=th, tol=v * 0.02, stencil="sw", omega=1.0)
    assert np.isfinite(b[0]).all()
    assert a[1:] == b[1:] and same_bits(a[0], b[0])
