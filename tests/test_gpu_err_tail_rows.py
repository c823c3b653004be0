"""The small error levels in one cluster launch, dealt by rows: held in the
cluster's shared memory, or in global memory where that does not fit, against
the oracle, bit for bit."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


# 10 x 10 x 645 over 5 x 5 x 323 (too large for shared memory), 10 x 10 x 150
# over 25 rows (CTAs without a row), 10 x 10 x 10 over 125 nodes, even and odd
# extents with three levels
@pytest.mark.parametrize("shape", [(20, 19, 1290), (19, 20, 299), (20, 20, 19), (74, 41, 39)])
def test_vcycle_rows(shape):
    from ion_gym_gb300.physics import multigrid3d as M
    rng = np.random.default_rng(shape[2])
    fixed = np.zeros(shape, bool)
    fixed[0] = fixed[:, -1] = True
    fixed |= rng.random(shape) < 0.003
    val = np.where(fixed, rng.uniform(-50, 50, shape), 0.0)
    a = M.solve3d_vmg(fixed, val, tol=1e-6)
    b = port.solve3d_vmg(fixed, val, tol=1e-6)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])
