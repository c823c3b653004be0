"""solve3d's resident loop, where nodes wait for their neighbours' versions
and the convergence test comes a pair late: the pair that met tol is the one
that is returned, at the first pair, the cap and in between, for shares of
slots at the edges of CTAs and rounds, on flat axes and with theta."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _deck(shape, seed):
    rng = np.random.default_rng(seed)
    fixed = rng.random(shape) < 0.02
    fixed[0, 0, 0] = True
    return fixed, np.where(fixed, rng.uniform(-100, 100, shape), 0.0)


# fewer slots than CTAs, one a CTA and one more (152, 153), a share of 1024
# and of 1025 slots, axes of one and two nodes
@pytest.mark.parametrize("shape", [(3, 3, 3), (1, 1, 305), (2, 2, 76), (1, 153, 2), (64, 32, 152),
                                   (61, 64, 80), (40, 1, 37), (2, 31, 2)])
@pytest.mark.parametrize("tol", [1e9, 0.5, 1e-6])
def test_stops_at_the_references_pair(shape, tol):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck(shape, 21)
    a = S.solve3d(fixed, val, tol=tol, omega=1.4)
    b = port.solve3d(fixed, val, tol=tol, omega=1.4)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])


@pytest.mark.parametrize("sweeps", [1, 2, 7])
def test_cap(sweeps):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck((20, 21, 22), 22)
    with pytest.raises(S.SolveNotConverged, match=f"cap of {sweeps} sweeps"):
        S.solve3d(fixed, val, tol=1e-300, max_sweeps=sweeps, omega=1.4)


@pytest.mark.parametrize("stencil", ["ghost_linear", "sw"])
@pytest.mark.parametrize("shape", [(9, 8, 7), (1, 40, 41), (62, 63, 81)])
def test_theta(shape, stencil):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck(shape, 23)
    rng = np.random.default_rng(24)
    theta = np.ones((6,) + shape, np.float32)
    cut = rng.random((6,) + shape) < 0.005
    theta[cut] = rng.uniform(0.2, 0.9, int(cut.sum())).astype(np.float32)
    a = S.solve3d(fixed, val, theta=theta, tol=1e-5, omega=1.0, stencil=stencil)
    b = port.solve3d(fixed, val, theta=theta, tol=1e-5, omega=1.0, stencil=stencil)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])


# a leg along an axis of one node is the node itself: its value of the pair
# before, also where most warps have cut nodes alone
@pytest.mark.parametrize("stencil", ["ghost_linear", "sw"])
@pytest.mark.parametrize("shape", [(1, 90, 91), (67, 1, 80), (75, 74, 1), (1, 1, 400), (1, 1, 1)])
def test_theta_on_axes_of_one_node(shape, stencil):
    from ion_gym_gb300.physics import solver3d as S
    fixed, val = _deck(shape, 25)
    rng = np.random.default_rng(26)
    theta = np.ones((6,) + shape, np.float32)
    cut = (rng.random(shape) < 0.09) & ~fixed
    theta[:, cut] = rng.uniform(0.3, 1.0, (6, int(cut.sum()))).astype(np.float32)
    a = S.solve3d(fixed, val, theta=theta, tol=1e-6, omega=1.0, stencil=stencil)
    b = port.solve3d(fixed, val, theta=theta, tol=1e-6, omega=1.0, stencil=stencil)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])
