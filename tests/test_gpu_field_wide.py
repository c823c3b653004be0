"""float64 fields of float32 potentials written directly (the composer's
default channel type) are the float32 fields widened, bit for bit: every
channel-group size, both spacing types, odd shapes, values that widen on
either path (zeros of both signs, subnormals, infinities, NaN); and a
superposition's last nodes past a float4 group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 8, 33), (17, 31, 29)])
def test_wide_fields(shape, nch):
    import torch
    from ion_gym_gb300.physics import field3d
    g = torch.Generator().manual_seed(nch * 100 + shape[0])
    phi = torch.randn((nch,) + shape, generator=g)
    phi[torch.rand(phi.shape, generator=g) < 0.1] = 0.0
    phi *= 2.0 ** torch.randint(-140, 20, phi.shape, generator=g).float()
    flat = phi.view(-1)
    flat[0], flat[3], flat[-1] = float("inf"), float("nan"), -0.0
    phi = phi.cuda()
    metal = torch.rand(shape, generator=g).cuda() < 0.3
    for h in (0.1, np.float64(0.1), 2.0 ** 30):
        narrow = torch.empty((3, nch) + shape, dtype=torch.float32, device="cuda")
        wide = torch.empty((3, nch) + shape, dtype=torch.float64, device="cuda")
        field3d._field_device(phi, metal, h, True, out=narrow)
        field3d._field_device(phi, metal, h, True, out=wide)
        a, b = wide.cpu().numpy(), narrow.double().cpu().numpy()
        nan = np.isnan(b)
        assert np.array_equal(np.isnan(a), nan)
        assert np.array_equal(a[~nan].view(np.int64), b[~nan].view(np.int64))


@pytest.mark.parametrize("n", [1, 3, 4, 7, 1021, 1024])
def test_superposition_tail(n):
    import torch
    from ion_gym_gb300.physics import field3d
    bases = field3d.padded(5, (1, 1, n))
    bases.copy_(torch.randn(bases.shape, generator=torch.Generator().manual_seed(n)))
    rows = np.array([0, 3, 4, 1])
    w = np.array([[0.5, -2.0, 3.0, 0.0], [1, 1, 1, 1]], np.float32)
    m = np.array([[1, 1, 1, 0], [0, 2, 1, 1]], np.uint8)
    got = field3d.superpose_device(bases, rows, w, m).cpu().numpy()
    b = bases.cpu().numpy()
    for c in range(2):
        acc = np.zeros((1, 1, n), np.float32)
        for s in range(4):
            for _ in range(m[c, s]):
                acc = acc + w[c, s] * b[rows[s]]
        assert np.array_equal(got[c].view(np.int32), acc.view(np.int32))


@pytest.mark.parametrize("h", [0.1, 3.0, 1.0 / 3.0, 2.0 ** -30, 1e-40, np.pi])
def test_float64_gradients(h):
    """float64 fields (divided by multiply-adds) are numpy's, over the whole
    exponent range: quotients near rounding boundaries, zeros of both signs,
    subnormals, infinities; every march length."""
    from ion_gym_gb300.physics.field3d import build_field_aware_3d
    for seed, shape in enumerate([(33, 33, 33), (5, 3, 2), (130, 9, 40), (2, 300, 290)]):
        rng = np.random.default_rng(seed)
        phi = rng.uniform(-1, 1, shape) * 2.0 ** rng.choice([0, 0, 0, 900, -900, -1060], shape)
        phi[rng.random(shape) < 0.1] = 0.0
        phi[rng.random(shape) < 0.05] = -0.0
        phi[rng.random(shape) < 0.2] = 0.25
        phi.flat[1] = np.inf
        with np.errstate(all="ignore"):
            want = np.gradient(phi, h)
        got = build_field_aware_3d(phi, np.zeros(shape, np.int16), h, electrode_aware=False)
        for g, w in zip(got, want):
            w = -w
            nan = np.isnan(w)
            assert np.array_equal(np.isnan(g), nan)
            assert np.array_equal(g[~nan].view(np.int64), w[~nan].view(np.int64))
