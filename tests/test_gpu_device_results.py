"""Mixed results written to device tensors by the kernel that forms them are
the host results, bit for bit: potentials and unit bases, tensors with an
offset, and what lies around them is left alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n_b", [((20, 21, 23), 1), ((17, 30, 33), 3)])
@pytest.mark.parametrize("unit", [False, True])
def test_device_out(shape, n_b, unit):
    import torch
    from ion_gym_gb300.physics.mixed import MixedSession
    rng = np.random.default_rng(n_b)
    masks = []
    for q in range(n_b):
        m = np.zeros(shape, bool)
        lo = [int(rng.integers(1, s - s // 3)) for s in shape]
        m[tuple(slice(a, a + 3) for a in lo)] = True
        masks.append(m)
    box = np.zeros(shape, bool)
    box[0] = box[-1] = True
    dt = torch.float32 if unit else torch.float64
    n = n_b * int(np.prod(shape))
    room = torch.full((n + 6,), -7.0, dtype=dt, device="cuda")
    out = room[3:3 + n].view((n_b,) + shape)
    with MixedSession(np.any(masks, 0) | box, n_b) as s:
        solve = s.solve_unit_bases if unit else s.solve_bases
        host = np.asarray(solve(masks, 1e4, 1e-9)).copy()
        solve(masks, 1e4, 1e-9, out=out)
    got = out.cpu().numpy()
    assert got.dtype == host.dtype and got.tobytes() == host.tobytes()
    assert bool((room[:3] == -7).all()) and bool((room[-3:] == -7).all())


@pytest.mark.parametrize("unit,shift", [(False, 4), (False, 1), (True, 2), (True, 1)])
def test_device_out_at_any_address(unit, shift):
    """A result at an address that its type is not aligned to is copied."""
    import torch
    from ion_gym_gb300.physics.mixed import MixedSession
    shape = (17, 19, 21)
    mask = np.zeros(shape, bool)
    mask[5:8, 6:9, 7:11] = True
    metal = mask.copy()
    metal[0] = metal[-1] = True
    n = int(np.prod(shape)) * (4 if unit else 8)
    room = torch.full((n + 16,), 99, dtype=torch.uint8, device="cuda")
    with MixedSession(metal, 1) as s:
        solve = s.solve_unit_bases if unit else s.solve_bases
        host = np.asarray(solve([mask], 1e4, 1e-9)).copy()
        solve([mask], 1e4, 1e-9, out=room[shift:shift + n])
    got = room.cpu().numpy()
    assert got[shift:shift + n].tobytes() == host.tobytes()
    assert (got[:shift] == 99).all() and (got[shift + n:] == 99).all()
