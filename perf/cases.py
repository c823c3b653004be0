"""The field solver's everyday calls, as cases to time.

A case is a dict of plain values; prepare() makes what a program holds before
the call, run() is one call through the public entry points, work() the bytes
and operations the call cannot do without, exact() the same outputs from
plain torch in 64 bits.

Kinds (sizes from this repository's benchmark and tests, or generic):

  sor        solver3d.solve3d on host arrays: one Dirichlet problem by
             red-black SOR, plain or with surface fractions (theta)
  door       multigrid3d.solve_bases_mg on host arrays: the FP64 basis door
             (V-cycle, one basis per electrode), plain or with theta
  cascadic   multigrid3d.solve3d_cascadic_relres on device arrays: the FP64
             cascadic solve of a quadrupole
  bases      MixedSession.solve_bases / solve_unit_bases: all bases of a deck
             in one batch on a resident session (ring stacks, planar boards)
  values     MixedSession.solve_values from pinned host buffers: one
             Dirichlet problem on a resident session
  decks      MixedSession.rebind + solve_values: a fresh batch of decks of
             one grid shape on the session the last batch left
  compose    field3d.compose_drive_channels on device bases: drive
             superposition and electrode-aware fields of all channels
  geometry   rasterize3d.rasterize + fractions_from_scene_device: a scene to
             its label grid and surface fractions
  field      field3d.build_field_aware_3d on host arrays: one potential's
             electrode-aware field
"""
import contextlib
import io
import math

import numpy as np
import torch

from ion_gym_gb300 import workloads
from ion_gym_gb300.physics import field3d, multigrid3d, rasterize3d, scene3d, solver3d
from ion_gym_gb300.physics.mixed import MixedSession

V_BASIS = 1e4      # the basis doors' default electrode voltage
ACCURACY = 1e-9    # of the electrode span: the mixed sessions' default


def listed():
    return [
        # one small drop-in solve: the reference's first example, a sphere-like
        # electrode in a grounded box; many short launches
        dict(name="sor_65", kind="sor", nx=65, ny=65, nz=65, theta=False,
             stencil="ghost_linear"),
        # the same call with surface fractions, the other stencil, odd sizes
        dict(name="sor_theta_sw", kind="sor", nx=57, ny=71, nz=90, theta=True,
             stencil="sw"),
        # the basis door as the reference's build calls it: every electrode
        dict(name="door_97", kind="door", nx=97, ny=97, nz=193, n=8, theta=False,
             stencil="ghost_linear"),
        # the basis door with surface fractions (scene-built decks)
        dict(name="door_theta", kind="door", nx=65, ny=65, nz=129, n=4, theta=True,
             stencil="ghost_linear"),
        # the benchmark's headline workload
        dict(name="cascadic_257", kind="cascadic", side=257),
        # the benchmark's ring stack: 8 bases in one batch, results on the device
        dict(name="bases_rings", kind="bases", deck="rings", nx=193, ny=193, nz=385, n=8,
             unit=False),
        # a served planar board: float32 unit bases for the field cache
        dict(name="bases_board", kind="bases", deck="board", nx=256, ny=64, nz=48, n=24,
             unit=True),
        # the benchmark's mixed quadrupole, from pinned host buffers
        dict(name="values_257", kind="values", side=257),
        # an uneven batch's share of one shape, small grids
        dict(name="decks_65", kind="decks", side=65, n=8),
        # the field build of the ring stack, default channel type
        dict(name="compose_rings", kind="compose", nx=193, ny=193, nz=385, n=8,
             channel_dtype="float64"),
        # a scene to masks and surface fractions, host results
        dict(name="geometry_97", kind="geometry", nx=97, ny=97, nz=193, n=8),
        # the smallest call: one potential's field on a small grid
        dict(name="field_33", kind="field", nx=33, ny=33, nz=33, dtype="float64"),
    ]


def _span(rng, lo, hi):
    """An integer spread over [lo, hi] by its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["sor", "door", "cascadic", "bases", "bases", "values", "decks",
                       "compose", "geometry", "field"])
    if kind == "sor":
        return dict(kind=kind, nx=_span(rng, 33, 97), ny=_span(rng, 33, 97),
                    nz=_span(rng, 33, 97), theta=rng.random() < 0.5,
                    stencil=rng.choice(["ghost_linear", "sw"]))
    if kind == "door":
        xy = _span(rng, 49, 97)
        return dict(kind=kind, nx=xy, ny=xy + rng.randint(-4, 0), nz=_span(rng, 65, 161),
                    n=rng.randint(2, 5), theta=rng.random() < 0.5, stencil="ghost_linear")
    if kind == "cascadic":
        return dict(kind=kind, side=_span(rng, 65, 241))
    if kind == "bases":
        if rng.random() < 0.5:
            xy = _span(rng, 65, 193)
            return dict(kind=kind, deck="rings", nx=xy, ny=xy + rng.randint(-5, 0),
                        nz=_span(rng, 97, 385), n=rng.randint(2, 8), unit=rng.random() < 0.5)
        return dict(kind=kind, deck="board", nx=_span(rng, 128, 512), ny=_span(rng, 48, 128),
                    nz=_span(rng, 40, 96), n=rng.randint(6, 24), unit=rng.random() < 0.5)
    if kind == "values":
        return dict(kind=kind, side=_span(rng, 65, 257))
    if kind == "decks":
        side = _span(rng, 33, 129)
        return dict(kind=kind, side=side, n=rng.randint(2, 16 if side <= 97 else 8))
    if kind == "compose":
        xy = _span(rng, 65, 193)
        return dict(kind=kind, nx=xy, ny=xy + rng.randint(-5, 0), nz=_span(rng, 97, 385),
                    n=rng.randint(2, 8), channel_dtype=rng.choice(["float32", "float64"]))
    if kind == "geometry":
        xy = _span(rng, 49, 129)
        return dict(kind=kind, nx=xy, ny=xy + rng.randint(-5, 0), nz=_span(rng, 65, 257),
                    n=rng.randint(2, 8))
    return dict(kind="field", nx=_span(rng, 17, 129), ny=_span(rng, 17, 129),
                nz=_span(rng, 17, 129), dtype=rng.choice(["float32", "float64"]))


# ------------------------------------------------------------ geometries
class Rings:
    """Coaxial rings along z (or, with one ring of inner radius 0, a solid
    cylinder) at real-valued radii and heights in a grounded box."""

    def __init__(self, shape, n, seed):
        rng = np.random.default_rng(seed)
        nx, ny, nz = shape
        self.shape = shape
        self.cx = (nx - 1) / 2.0 + rng.uniform(-0.4, 0.4)
        self.cy = (ny - 1) / 2.0 + rng.uniform(-0.4, 0.4)
        m = min(nx, ny)
        pitch = (nz - 6) / n
        self.rings = []
        for e in range(n):
            r = rng.uniform(0.12, 0.30) * m
            t = rng.uniform(2.6, 0.42 * pitch) if 0.42 * pitch > 2.6 else 2.2
            z = 3 + e * pitch + rng.uniform(0.1, 0.3) * pitch
            self.rings.append((r, r + rng.uniform(2.8, 4.6), z, z + t))
        if n == 1:
            r = rng.uniform(0.14, 0.18) * m
            z = rng.uniform(0.36, 0.42) * nz
            self.rings = [(0.0, r, z, z + rng.uniform(0.2, 0.26) * nz)]

    def inside(self, e, x, y, z):
        """Points in ring e: within its outer cylinder (surface included),
        not strictly within its bore."""
        lo, hi, za, zb = self.rings[e]
        rr = (x - self.cx) ** 2 + (y - self.cy) ** 2
        return (rr <= hi * hi) & (rr >= lo * lo) & (z >= za) & (z <= zb)

    def grid(self):
        return torch.meshgrid(*(torch.arange(s, dtype=torch.float64, device="cuda")
                                for s in self.shape), indexing="ij")

    def masks(self):
        """{1..n: CUDA bool} and the grounded box."""
        g = self.grid()
        box = torch.zeros(self.shape, dtype=torch.bool, device="cuda")
        for a in range(3):
            box.select(a, 0).fill_(True)
            box.select(a, self.shape[a] - 1).fill_(True)
        return {e + 1: self.inside(e, *g) & ~box for e in range(len(self.rings))}, box

    def theta(self, metal):
        """(6, nx, ny, nz) float32: the fraction of each metal-facing leg to
        the ring's surface, by bisection."""
        th = torch.ones((6,) + self.shape, dtype=torch.float32, device="cuda")
        for d in range(6):
            a, step = d // 2, (-1, 1)[d & 1]
            near = torch.roll(metal, -step, a)
            near.select(a, 0 if step < 0 else self.shape[a] - 1).fill_(False)
            legs = (near & ~metal).nonzero()
            org = legs.to(torch.float64)
            lo = torch.zeros(len(legs), dtype=torch.float64, device="cuda")
            hi = torch.ones_like(lo)
            for _ in range(45):
                mid = 0.5 * (lo + hi)
                p = org.clone()
                p[:, a] += step * mid
                hit = torch.zeros(len(legs), dtype=torch.bool, device="cuda")
                for e in range(len(self.rings)):
                    hit |= self.inside(e, p[:, 0], p[:, 1], p[:, 2])
                hi = torch.where(hit, mid, hi)
                lo = torch.where(hit, lo, mid)
            th[d][tuple(legs.T)] = (0.5 * (lo + hi)).clamp(1e-3, 1.0).to(torch.float32)
        return th

    def scene(self):
        els = []
        for e, (lo, hi, za, zb) in enumerate(self.rings):
            bore = scene3d.Cylinder(self.cx, self.cy, zb + 1.0, lo, zb - za + 2.0)
            out = scene3d.Cylinder(self.cx, self.cy, zb, hi, zb - za)
            els.append(scene3d.Electrode(e + 1, f"ring{e + 1}",
                                         [scene3d.Shape([out], [bore])]))
        return scene3d.GeomScene(scene3d.GridSpec(*self.shape), els)


def _shape(c):
    return (c["nx"], c["ny"], c["nz"])


def _deck(c, seed):
    """A bases case's masks (n, nx, ny, nz) and metal, host bool arrays."""
    shape = _shape(c)
    if c["deck"] == "rings":
        n, nz, m = c["n"], shape[2], min(shape[:2])
        room = max(2.0, (nz - 8 - 4 * n) / max(1, n - 1))
        masks, box = workloads.ring_stack(seed, shape, n, 4, 0.1 * m, 0.31 * m,
                                          max(1, int(0.2 * room)), max(2, int(0.6 * room)))
    else:
        # thin polygons can miss every node: the first n that do not
        masks, box = workloads.planar_board(seed, shape, 2 * c["n"])
        masks = dict(sorted((k, m) for k, m in masks.items() if (m & ~box).any())[:c["n"]])
    stack = np.stack([masks[k] & ~box for k in sorted(masks)])
    return stack, stack.any(0) | box


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _potentials(shape, count, seed):
    """Smooth device potentials in [0, 1] like unit bases."""
    rng = np.random.default_rng(seed)
    ax = [torch.linspace(-1, 1, s, dtype=torch.float64, device="cuda") for s in shape]
    out = []
    for _ in range(count):
        f = 1.0
        for a in range(3):
            g = torch.exp(-((ax[a] - rng.uniform(-0.6, 0.6)) / rng.uniform(0.3, 0.9)) ** 2)
            f = f * g.reshape([-1 if b == a else 1 for b in range(3)])
        out.append(f)
    return out


# ------------------------------------------------------------ cases
def _sor_inputs(c, seed):
    r = Rings(_shape(c), 1, seed)
    masks, box = r.masks()
    v = 50.0 + 100.0 * np.random.default_rng(seed + 1).random()
    fixed = masks[1] | box
    return fixed, masks[1].to(torch.float64) * v, r.theta(fixed) if c["theta"] else None


def _door_inputs(c, seed):
    r = Rings(_shape(c), c["n"], seed)
    masks, box = r.masks()
    metal = box.clone()
    for m in masks.values():
        metal |= m
    return masks, box, metal, r.theta(metal) if c["theta"] else None


def _compose_inputs(c, seed):
    r = Rings(_shape(c), c["n"], seed)
    masks, box = r.masks()
    label = torch.zeros(_shape(c), dtype=torch.int16, device="cuda")
    metal = box.clone()
    for e, m in masks.items():
        label[m] = e
        metal |= m
    bases = {}
    for e, f in enumerate(_potentials(_shape(c), c["n"], seed), 1):
        f = torch.where(metal, masks[e].to(f.dtype), f)
        bases[e] = f.to(torch.float32)
    label[box] = c["n"] + 1
    spec = workloads.ring_stack_drive(c["n"], 0.1, seed)
    spec.geometry.channel_dtype = c["channel_dtype"]
    return spec, bases, label


def _field_inputs(c, seed):
    r = Rings(_shape(c), 1, seed)
    masks, box = r.masks()
    phi = _potentials(_shape(c), 1, seed)[0] * 100.0
    phi = torch.where(box, torch.zeros_like(phi), torch.where(masks[1], 100.0, phi))
    return phi.to(getattr(torch, c["dtype"])), (masks[1] | box)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind, "case": c}
    if kind == "sor":
        fixed, val, th = _sor_inputs(c, seed)
        s.update(fixed=fixed.cpu().numpy(), val=val.cpu().numpy(),
                 theta=None if th is None else th.cpu().numpy())
    elif kind == "door":
        masks, box, metal, th = _door_inputs(c, seed)
        s["masks"] = {e: m.cpu().numpy() for e, m in masks.items()}
        s["masks"][c["n"] + 1] = box.cpu().numpy()
        s.update(only=set(masks), theta=None if th is None else th.cpu().numpy())
    elif kind == "cascadic":
        fixed, val = _quadrupole(c["side"], seed)
        s.update(fixed=torch.from_numpy(fixed).cuda().to(torch.uint8),
                 val=torch.from_numpy(val).cuda())
        s["out"] = torch.empty_like(s["val"])
    elif kind == "bases":
        stack, metal = _deck(c, seed)
        n = len(stack)
        s["session"] = MixedSession(metal, n)
        s["masks"] = torch.from_numpy(stack.view(np.uint8)).cuda()
        if c["unit"]:   # the field cache's float32 arrays live on the host
            s["out"] = torch.empty(stack.shape, dtype=torch.float32).pin_memory().numpy()
        else:
            s["out"] = torch.empty(stack.shape, dtype=torch.float64, device="cuda")
    elif kind == "values":
        fixed, val = _quadrupole(c["side"], seed)
        s.update(session=MixedSession(fixed, 1), val=_pinned(val[None]), span=2.0 * val.max())
        s["out"] = _pinned(np.empty_like(s["val"]))
    elif kind == "decks":
        pairs = [_random_deck(c, seed, q) for q in range(c["n"])]
        s["metals"] = np.stack([f for f, _ in pairs])
        s["val"] = _pinned(np.stack([v for _, v in pairs]))
        s["spans"] = [float(np.ptp(v)) for _, v in pairs]
        s["out"] = _pinned(np.empty_like(s["val"]))
        s["session"] = MixedSession(s["metals"])
    elif kind == "compose":
        s["spec"], s["bases"], s["label"] = _compose_inputs(c, seed)
    elif kind == "geometry":
        s["scene"] = Rings(_shape(c), c["n"], seed).scene()
    else:
        phi, metal = _field_inputs(c, seed)
        s.update(phi=phi.cpu().numpy(), label=metal.cpu().numpy().astype(np.int16))
    return s


def _quadrupole(side, seed):
    rng = np.random.default_rng(seed)
    return workloads.quadrupole(side, side * rng.uniform(0.115, 0.13), rng.uniform(0.8, 1.2))


def _random_deck(c, seed, q):
    return workloads.random_deck(1000 * seed + q, c["side"], 2 + q % 15)


def run(state):
    s, kind = state, state["kind"]
    if kind == "sor":
        return list(solver3d.solve3d(s["fixed"], s["val"], theta=s["theta"], tol=1e-7,
                                     stencil=s["case"]["stencil"]))
    if kind == "door":
        with contextlib.redirect_stdout(io.StringIO()):   # the door's progress lines
            out = multigrid3d.solve_bases_mg(s["masks"], v_basis=V_BASIS, tol=1e-5,
                                             theta=s["theta"], only=s["only"],
                                             stencil=s["case"]["stencil"])
        return {str(e): phi for e, phi in out.items()}
    if kind == "cascadic":
        return list(multigrid3d.solve3d_cascadic_relres(s["fixed"], s["val"], out=s["out"]))
    if kind == "bases":
        solve = (s["session"].solve_unit_bases if s["case"]["unit"]
                 else s["session"].solve_bases)
        return solve(s["masks"], V_BASIS, ACCURACY, out=s["out"])
    if kind == "values":
        return s["session"].solve_values(s["val"], ACCURACY, out=s["out"], span=s["span"])
    if kind == "decks":
        s["session"].rebind(s["metals"])
        return s["session"].solve_values(s["val"], ACCURACY, out=s["out"], span=s["spans"])
    if kind == "compose":
        r = field3d.compose_drive_channels(s["spec"], s["bases"], s["label"])
        return {k: v for k, v in r.items() if k != "ch_name"}
    if kind == "geometry":
        label = rasterize3d.rasterize(s["scene"])
        return [label, rasterize3d.fractions_from_scene_device(s["scene"], label > 0)]
    return list(field3d.build_field_aware_3d(s["phi"], s["label"], 0.1))


def work(case):
    """Inputs read once, outputs written once; operations of the least the
    method named can do (a sweep pair is 8 per node)."""
    c, kind = case, case["kind"]
    n = float(c["side"] ** 3 if "side" in c else c["nx"] * c["ny"] * c["nz"])
    long = c.get("side") or max(c["nx"], c["ny"], c["nz"])
    if kind == "sor":
        return {"bytes": n * (17 + (24 if c["theta"] else 0)), "flops": 8 * n * 2.5 * long}
    if kind == "door":
        return {"bytes": c["n"] * n * 10 + (24 * n if c["theta"] else 0),
                "flops": c["n"] * n * 8 * 90}
    if kind == "cascadic":
        return {"bytes": n * 17, "flops": 8 * n * 6.0 * long}
    if kind == "bases":
        return {"bytes": c["n"] * n * (5 if c["unit"] else 9), "flops": c["n"] * n * 8 * 40}
    if kind == "values":
        return {"bytes": n * 16, "flops": n * 8 * 40}
    if kind == "decks":
        return {"bytes": c["n"] * n * 17, "flops": c["n"] * n * 8 * 40}
    if kind == "compose":
        per = 8 if c["channel_dtype"] == "float64" else 4
        ch = 4   # static, two phases, the gate
        return {"bytes": n * (4 * c["n"] + 2 + 4 * (ch - 1) + 3 * per * ch),
                "flops": n * (2 * c["n"] + 6) * ch}
    if kind == "geometry":
        return {"bytes": n * (2 + 1 + 24), "flops": n * 8 * c["n"]}
    per = 8 if c["dtype"] == "float64" else 4
    return {"bytes": n * (4 * per + 1), "flops": n * 6}


# ------------------------------------------------------------ 64-bit values
def _tight(fixed, val, theta=None, stencil="ghost_linear", rel=1e-13):
    """The discrete Dirichlet solution by red-black SOR with over-relaxation
    (every neighbour rule of the operator; reflecting faces)."""
    shape = fixed.shape
    free = ~fixed
    u = torch.where(fixed, val, torch.zeros_like(val))
    if theta is None:
        w, den = [1.0] * 6, torch.full_like(u, 6.0)
    else:
        t = theta.to(torch.float64)
        if stencil == "sw":
            w = [1.0 / (t[d] * (t[d] + t[d ^ 1])) for d in range(6)]
        else:
            w = [1.0 / t[d] for d in range(6)]
        den = sum(w)
    idx = torch.meshgrid(*(torch.arange(s, device="cuda") for s in shape), indexing="ij")
    red = (idx[0] + idx[1] + idx[2]) % 2 == 0
    half = [free & red, free & ~red]
    rho = sum(math.cos(math.pi / (s + 1)) for s in shape) / 3.0
    om = 2.0 / (1.0 + math.sqrt(1.0 - rho * rho))
    span = float(val.abs().max())
    for it in range(40 * max(shape)):
        before = u
        for h in half:
            p = torch.nn.functional.pad(u[None, None], (1,) * 6, mode="reflect")[0, 0]
            c = slice(1, -1)
            q = (w[0] * p[:-2, c, c] + w[1] * p[2:, c, c] + w[2] * p[c, :-2, c]
                 + w[3] * p[c, 2:, c] + w[4] * p[c, c, :-2] + w[5] * p[c, c, 2:]) / den
            u = torch.where(h, u + om * (q - u), u)
        if it % 25 == 24 and float((u - before).abs().max()) < rel * span:
            break
    return u


def _tight_cg(fixed, val, rel=1e-12):
    """The same for a grounded box with theta None, by conjugate gradients
    (the box faces are fixed, so the operator is symmetric)."""
    c = slice(1, -1)
    free = (~fixed)[c, c, c].to(torch.float64)

    def lap(p):   # (6 - neighbours) p on the interior
        r = 6.0 * p[c, c, c]
        for a in (p[:-2, c, c], p[2:, c, c], p[c, :-2, c], p[c, 2:, c], p[c, c, :-2],
                  p[c, c, 2:]):
            r -= a
        return r.mul_(free)

    u = torch.where(fixed, val, torch.zeros_like(val))
    r = -lap(u)
    p = torch.zeros_like(u)
    p[c, c, c] = r
    rr = (r * r).sum()
    stop = float(rr) * rel * rel
    for it in range(6000):
        q = lap(p)
        pi = p[c, c, c]
        a = rr / (pi * q).sum()
        u[c, c, c].addcmul_(pi, a)
        r.addcmul_(q, -a)
        new = (r * r).sum()
        pi.mul_(new / rr).add_(r)
        rr = new
        if it % 50 == 49 and float(rr) < stop:
            break
    return u


def _grad(phi, metal, h):
    """-numpy.gradient, one-sided into the vacuum at metal nodes with vacuum
    on exactly one side along an axis."""
    out = []
    for a in range(3):
        n = phi.shape[a]
        d = torch.empty_like(phi)
        up, dn = phi.narrow(a, 1, n - 1), phi.narrow(a, 0, n - 1)
        step = (up - dn) / h                      # step i: nodes i -> i + 1
        d.narrow(a, 1, n - 2).copy_((phi.narrow(a, 2, n - 2) - phi.narrow(a, 0, n - 2)) / (2 * h))
        d.select(a, 0).copy_(step.select(a, 0))
        d.select(a, n - 1).copy_(step.select(a, n - 2))
        vac_up = torch.zeros_like(metal)
        vac_dn = torch.zeros_like(metal)
        vac_up.narrow(a, 0, n - 1).copy_(~metal.narrow(a, 1, n - 1))
        vac_dn.narrow(a, 1, n - 1).copy_(~metal.narrow(a, 0, n - 1))
        pad = step.new_zeros(step.select(a, 0).unsqueeze(a).shape)
        fwd, bwd = torch.cat([step, pad], a), torch.cat([pad, step], a)
        d = torch.where(metal & vac_up & ~vac_dn, fwd, d)
        d = torch.where(metal & vac_dn & ~vac_up, bwd, d)
        out.append(-d)
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "sor":
        fixed, val, th = _sor_inputs(c, seed)
        return [_tight(fixed, val, th, c["stencil"]), None, None]
    if kind == "door":
        masks, box, metal, th = _door_inputs(c, seed)
        solve = _tight_cg if th is None else (lambda f, v: _tight(f, v, th, c["stencil"]))
        return {str(e): solve(metal, m.to(torch.float64) * V_BASIS) for e, m in masks.items()}
    if kind == "cascadic":
        fixed, val = _quadrupole(c["side"], seed)
        return [_tight_cg(torch.from_numpy(fixed).cuda(), torch.from_numpy(val).cuda()),
                None, None, None]
    if kind == "bases":
        stack, metal = _deck(c, seed)
        metal = torch.from_numpy(metal).cuda()
        v = 1.0 if c["unit"] else V_BASIS
        return torch.stack([_tight_cg(metal, torch.from_numpy(m).cuda().to(torch.float64) * v)
                            for m in stack])
    if kind == "values":
        fixed, val = _quadrupole(c["side"], seed)
        return _tight_cg(torch.from_numpy(fixed).cuda(), torch.from_numpy(val).cuda())[None]
    if kind == "decks":
        return torch.stack([_tight_cg(torch.from_numpy(f).cuda(), torch.from_numpy(v).cuda())
                            for f, v in (_random_deck(c, seed, q) for q in range(c["n"]))])
    if kind == "compose":
        spec, bases, label = _compose_inputs(c, seed)
        els = spec.geometry.electrodes
        names = [g.name for g in spec.geometry.rf_groups]
        pots = [sum(bases[e].to(torch.float64) * float(np.float32(el.dc))
                    for e, el in enumerate(els, 1))]
        used = [nm for nm in names if any(nm in el.group_names() for el in els)]
        pots += [sum(bases[e].to(torch.float64) for e, el in enumerate(els, 1)
                     if nm in el.group_names()) for nm in used]
        g = [_grad(p, label != 0, 0.1) for p in pots]
        out = {k: g[0][a] for a, k in enumerate(("EAx", "EAy", "EAz"))}
        out.update({k: torch.stack([x[a] for x in g[1:]])
                    for a, k in enumerate(("ExK", "EyK", "EzK"))})
        out["chan_phi"] = pots[1:]
        return out
    if kind == "geometry":
        r = Rings(_shape(c), c["n"], seed)
        metal = torch.zeros(_shape(c), dtype=torch.bool, device="cuda")
        g = r.grid()
        for e in range(c["n"]):
            metal |= r.inside(e, *g)
        return [None, r.theta(metal).to(torch.float64)]
    phi, metal = _field_inputs(c, seed)
    return _grad(phi.to(torch.float64), metal, 0.1)
