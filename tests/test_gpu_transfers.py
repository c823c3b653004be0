"""The V-cycle's transfers and bottom solve against the oracle, bit for bit:
restriction by fused multiply-adds and the trilinear value by sums, on
values whose weighted products would round (subnormals), cancel, are zeros
of either sign, infinite or NaN, and on shapes whose coarse grid clamps; the
one-CTA bottom through whole V-cycles whose bottoms have one node per
thread, several, and more than fit in shared memory."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import port

pytestmark = pytest.mark.gpu


def _values(rng, shape, special):
    v = rng.uniform(-1, 1, shape) * 2.0 ** rng.integers(-6, 7, shape)
    v[rng.random(shape) < 0.2] = 0.0
    if special == "tiny":
        v *= 2.0 ** rng.choice([-1073, -1060, -1020, -960, 0], shape)
    elif special == "huge":
        v *= 2.0 ** rng.choice([1016, 1010, 0], shape)
    elif special == "signed":
        v = np.where(rng.random(shape) < 0.4, -0.0, v)
        v[rng.random(shape) < 0.2] = 0.5
        v[rng.random(shape) < 0.2] = -0.5
    elif special == "nonfinite":
        v.flat[rng.integers(0, v.size, 3)] = [np.inf, -np.inf, np.nan]
    return v


def _same(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and same_bits(a[~nan], b[~nan])


SHAPES = [(17, 18, 33), (2, 3, 4), (1, 5, 8), (1, 1, 9), (9, 1, 2), (34, 33, 17)]


@pytest.mark.parametrize("special", ["", "tiny", "huge", "signed", "nonfinite"])
@pytest.mark.parametrize("shape", SHAPES)
def test_transfers(shape, special):
    from ion_gym_gb300.physics import _device as D
    rng = np.random.default_rng(sum(shape) + len(special))
    fine = _values(rng, shape, special)
    cs = tuple((s + 1) // 2 for s in shape)
    a, b = np.empty(cs), np.empty(cs)
    D.restrict_fw(fine, a)
    with np.errstate(all="ignore"):
        port.restrict_fw(fine, b)
    assert _same(a, b)
    fixed = rng.random(shape) < 0.2
    for c in (cs, tuple(max(1, s - 1) for s in cs)):   # the second clamps
        coarse = _values(rng, c, special)
        base = _values(rng, shape, "signed")
        a, b = base.copy(), base.copy()
        D.prolong_add(coarse, a, fixed)
        port.prolong_add(coarse, b, fixed)
        assert _same(a, b)
        assert _same(D.prolongate(coarse, shape), port.prolongate(coarse, shape))


# the bottom levels: 9 x 9 x 9 (one node a thread), 9 x 33 x 33 = 9801 (ten),
# 9 x 41 x 41 = 15129 (the launched loop)
@pytest.mark.parametrize("shape", [(17, 18, 17), (17, 65, 65), (18, 81, 82)])
def test_vcycle_bottoms(shape):
    from ion_gym_gb300.physics import multigrid3d as M
    rng = np.random.default_rng(shape[1])
    fixed = rng.random(shape) < 0.01
    fixed[0] = fixed[-1] = True
    val = np.where(fixed, rng.uniform(-50, 50, shape), 0.0)
    a = M.solve3d_vmg(fixed, val, tol=1e-7)
    b = port.solve3d_vmg(fixed, val, tol=1e-7)
    assert a[1:] == b[1:] and same_bits(a[0], b[0])


# levels that run below one launch: the first error level itself (33^3 and
# flat ones), a level below a launched one (49 x 49 x 49 under 97^3), two and
# three levels deep, single-node axes, theta
@pytest.mark.parametrize("shape", [(65, 66, 64), (97, 96, 95), (33, 35, 21), (20, 90, 140),
                                   (21, 19, 250)])
def test_vcycle_tails(shape):
    from ion_gym_gb300.physics import multigrid3d as M
    rng = np.random.default_rng(shape[2])
    fixed = np.zeros(shape, bool)
    fixed[:, 0] = fixed[:, -1] = True
    fixed |= rng.random(shape) < 0.002
    val = np.where(fixed, rng.uniform(-50, 50, shape), 0.0)
    for stencil in ("ghost_linear", "sw"):
        a = M.solve3d_vmg(fixed, val, tol=1e-6, stencil=stencil)
        b = port.solve3d_vmg(fixed, val, tol=1e-6, stencil=stencil)
        assert a[1:] == b[1:] and same_bits(a[0], b[0])


def test_tails_side_by_side():
    """Bases solved at once, each with its own cluster launches, keep the
    bits of one at a time."""
    from ion_gym_gb300.physics import multigrid3d as M
    from ion_gym_gb300.workloads import ring_stack
    masks, box = ring_stack(3, (65, 65, 129), 8, r_lo=8, r_hi=20, gap_lo=3, gap_hi=9)
    masks[9] = box
    many = M.solve_bases_mg(masks, tol=1e-5, only=set(range(1, 9)))
    one = M.solve_bases_mg(masks, tol=1e-5, only={4})
    ref = port.solve_bases_mg(masks, tol=1e-5, only={4, 7})
    assert same_bits(many[4], one[4])
    for e in (4, 7):
        assert same_bits(many[e], ref[e])
