"""float32 gradients whose nodes mix ordinary differences with the cases that
are taken apart (differences of -0, subnormal, huge, infinite or NaN; spacings
outside the fast divisions' range) are numpy's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [0.1, 3.0, 2.0 ** 30, 1e-30])
@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 11, 33), (20, 3, 65)])
def test_mixed_nodes(shape, h):
    from ion_gym_gb300.physics.field3d import build_field_aware_3d
    rng = np.random.default_rng(shape[2])
    phi = rng.uniform(-1, 1, shape) * 2.0 ** rng.choice([0, 0, 0, 0, 110, -110, -140], shape)
    phi = phi.astype(np.float32)
    phi[rng.random(shape) < 0.2] = 0.0
    phi[rng.random(shape) < 0.1] = -0.0
    phi[rng.random(shape) < 0.2] = 0.25
    phi.flat[1], phi.flat[-1] = np.inf, np.nan
    with np.errstate(all="ignore"):
        want = np.gradient(phi, h)
    got = build_field_aware_3d(phi, np.zeros(shape, np.int16), h, electrode_aware=False)
    for a in range(3):
        w = -want[a]
        g = np.asarray(got[a])
        assert w.dtype == np.float32
        nan = np.isnan(w)
        assert np.array_equal(np.isnan(g), nan)
        assert np.array_equal(g.astype(np.float32)[~nan].view(np.int32), w[~nan].view(np.int32))
