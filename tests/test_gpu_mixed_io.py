"""The mixed sessions' conversions in and out of the fixed point: unit bases
equal the float64 potentials divided and rounded on the host, bit for bit,
for voltages of every kind of significand and size; float64 potentials keep
the Dirichlet values exactly; node counts that do not fill a thread's four
nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _masks(shape):
    a, b = np.zeros(shape, bool), np.zeros(shape, bool)
    a[1:3, 1:4, 1:6] = True
    b[-4:-2, 2:5, -5:-1] = True
    return a, b


@pytest.mark.parametrize("v", [1e4, 1.0, -1e4, 3.0, 0.1, 1e-10, 7e15, -1.9999999999])
@pytest.mark.parametrize("shape", [(13, 12, 11), (9, 8, 33)])
def test_unit_bases(shape, v):
    from ion_gym_gb300.physics.mixed import MixedSession
    masks = _masks(shape)
    with MixedSession(masks[0] | masks[1], 2) as s:
        phi = s.solve_bases(masks, v)
        unit = s.solve_unit_bases(masks, v)
    want = (phi / v).astype(np.float32)
    assert np.array_equal(unit.view(np.int32), want.view(np.int32))
    for m, p in zip(masks, phi):
        assert np.all(p[m] == v) and np.all(p[(masks[0] | masks[1]) & ~m] == 0)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -40, 2.0 ** 59, 1.0 / 3.0])
def test_values(scale):
    from ion_gym_gb300.physics import multigrid3d as M
    from ion_gym_gb300.physics.mixed import MixedSession
    rng = np.random.default_rng(4)
    shape = (17, 15, 21)
    fixed = rng.random(shape) < 0.05
    fixed[0] = True
    val = np.where(fixed, rng.uniform(-1, 1, shape), 0.0) * scale
    with MixedSession(fixed, 1) as s:
        got = s.solve_values(val[None], accuracy=1e-9 * scale, span=1.0)[0]
    assert np.array_equal(got[fixed], val[fixed])
    ref = M.solve3d_vmg(fixed, val, tol=1e-13 * scale, max_cycles=200, accept_stagnation=True)[0]
    assert np.abs(got - ref).max() <= 2e-9 * scale
