"""The sweeps that give a thread two x-planes and the column residual
(single-kernel entry points, bit for bit against the oracle) at the edges of
their tiles: odd and even plane counts, one plane, reflecting and flat
faces, values with exact ties, zeros of both signs, subnormals and
infinities among them."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _values(rng, shape):
    v = rng.uniform(-1, 1, shape) * 2.0 ** rng.integers(-3, 4, shape)
    few = rng.random(shape)
    v[few < 0.1] = np.round(v[few < 0.1] * 8) / 8     # halves and zeros
    v[(few > 0.1) & (few < 0.13)] *= 2.0 ** -1060     # subnormal
    v[(few > 0.13) & (few < 0.15)] = -0.0
    return v


# 2 planes a thread from 622,592 slots of one colour on: 87 x 120 x 121 is
# over it, 85 x 120 x 121 under
@pytest.mark.parametrize("shape", [(87, 120, 121), (85, 120, 121), (1, 1201, 1100),
                                   (2, 900, 700), (5, 3, 4), (4, 1, 9), (3, 7, 1)])
@pytest.mark.parametrize("omega", [1.0, 1.85])
def test_sweeps(shape, omega):
    from ion_gym_gb300.physics import _device as D
    rng = np.random.default_rng(sum(shape))
    fixed = rng.random(shape) < 0.2
    for colour in (0, 1):
        a, b = (_values(np.random.default_rng(7 + colour), shape) for _ in range(2))
        da = D.sweep(a, fixed, None, omega, colour, True)
        db = port.sweep(b, fixed, np.ones((6,) + shape, np.float32), omega, colour, True)
        assert same_bits(a, b) and da == db
        f = _values(rng, shape)
        a, b = (_values(np.random.default_rng(9 + colour), shape) for _ in range(2))
        da = D.sweep_rhs(a, fixed, f, omega, colour)
        db = port.sweep_rhs(b, fixed, f, omega, colour)
        assert same_bits(a, b) and da == db


@pytest.mark.parametrize("shape", [(1, 5, 6), (2, 5, 6), (3, 4, 5), (4, 4, 5), (5, 33, 17),
                                   (6, 1, 40), (7, 20, 1), (41, 22, 19)])
def test_residuals(shape):
    from ion_gym_gb300.physics import _device as D
    rng = np.random.default_rng(sum(shape))
    phi, fixed = _values(rng, shape), rng.random(shape) < 0.2
    phi.flat[shape[2] // 2] = np.inf
    ones = np.ones((6,) + shape, np.float32)
    cut = np.where(rng.random(ones.shape) < 0.3, rng.uniform(0.2, 1, ones.shape), 1.0)
    for th in (None, cut.astype(np.float32)):
        for ghost in (True, False):
            a, b = np.full(shape, 7.0), np.full(shape, 7.0)
            D.residual(phi, fixed, th, ghost, a)
            port.residual(phi, fixed, ones if th is None else th, ghost, b)
            nan = np.isnan(b)
            assert np.array_equal(np.isnan(a), nan) and same_bits(a[~nan], b[~nan])
    e, f = _values(rng, shape), _values(rng, shape)
    a, b = np.full(shape, 7.0), np.full(shape, 7.0)
    D.residual_rhs(e, fixed, f, a)
    port.residual_rhs(e, fixed, f, b)
    assert same_bits(a, b)
