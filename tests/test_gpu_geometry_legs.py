"""The raster's integer node bounds and the theta kernel's per-leg primitive
lists against plain numpy in float64: bounds on, just inside and just
outside node planes, primitives off the grid, shapes with holes, more
primitives around one leg than a list holds, mirror planes, grids that do
not fill a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(rng, shape, n_el, crowd):
    from ion_gym_gb300.physics.scene3d import (Box3D, Cylinder, Electrode, GeomScene, GridSpec,
                                               Shape)
    els = []
    for e in range(n_el):
        shapes = []
        for _ in range(crowd):
            c = [rng.uniform(0, s) for s in shape]
            if rng.random() < 0.5:
                r = rng.choice([2.0, 3.0, 2.5, 5 ** 0.5, rng.uniform(1, 4)])
                c[:2] = [np.round(c[0]), np.round(c[1])] if rng.random() < 0.5 else c[:2]
                z = rng.choice([np.round(c[2]), np.round(c[2]) + 1e-9, c[2]])
                a = Cylinder(c[0], c[1], z, r, rng.choice([2.0, rng.uniform(1, 6)]))
                hole = Cylinder(c[0], c[1], z + 1, r * 0.6, 20.0)
            else:
                lo = [np.round(v) + rng.choice([0.0, 1e-9, -1e-9, 0.3]) for v in c]
                d = [rng.choice([1.0, 2.0, rng.uniform(0.5, 5)]) for _ in range(3)]
                a = Box3D(*lo, *[p + q for p, q in zip(lo, d)])
                hole = Box3D(lo[0] + 0.5, lo[1] - 9, lo[2] - 9, lo[0] + 1.0, lo[1] + 9, lo[2] + 9)
            shapes.append(Shape([a], [hole] if rng.random() < 0.4 else []))
        els.append(Electrode(e + 1, f"e{e + 1}", shapes))
    return GeomScene(GridSpec(*shape), els)


def _numpy_labels(scene, shape):
    from ion_gym_gb300.physics.rasterize3d import primitive_table
    table, idx, _ = primitive_table(scene)
    x, y, z = np.meshgrid(*(np.arange(s, dtype=float) for s in shape), indexing="ij")
    lab = np.zeros(shape, np.int16)
    clash = False
    for slot in range(len(idx)):
        m = np.zeros(shape, bool)
        rows = table[table[:, 1] == slot]
        for sid in np.unique(rows[:, 2]):
            w = np.zeros(shape, bool)
            for r in rows[rows[:, 2] == sid]:
                b = r[4:10]
                if r[0] == 0.0:
                    hit = (((x - b[0]) * (x - b[0]) + (y - b[1]) * (y - b[1]) <= b[2])
                           & (z >= b[3]) & (z <= b[4]))
                else:
                    hit = ((x >= b[0]) & (x <= b[1]) & (y >= b[2]) & (y <= b[3])
                           & (z >= b[4]) & (z <= b[5]))
                w = (w | hit) if r[3] == 0.0 else (w & ~hit)
            m |= w
        clash |= bool((m & (lab != 0)).any())
        lab[m] = idx[slot]
    return lab, clash


@pytest.mark.parametrize("seed", range(6))
def test_labels(seed):
    from ion_gym_gb300.physics.rasterize3d import rasterize
    rng = np.random.default_rng(seed)
    shape = ((19, 17, 23), (7, 40, 9), (33, 5, 31))[seed % 3]
    sc = _scene(rng, shape, 1 + seed % 2, 3)
    want, clash = _numpy_labels(sc, shape)
    if clash:
        with pytest.raises(ValueError, match="overlaps"):
            rasterize(sc)
    elif not all((want == e.index).any() for e in sc.electrodes):
        with pytest.raises(ValueError, match="EMPTY"):
            rasterize(sc)
    else:
        assert np.array_equal(rasterize(sc), want)


@pytest.mark.parametrize("mirror", [(False, False, False), (True, False, True)])
@pytest.mark.parametrize("seed,crowd", [(0, 2), (1, 5), (2, 40), (3, 12)])
def test_theta(seed, crowd, mirror):
    from ion_gym_gb300.physics import solver3d
    from ion_gym_gb300.physics.rasterize3d import fractions_from_scene_device
    rng = np.random.default_rng(100 + seed)
    shape = ((19, 17, 23), (7, 12, 9), (33, 5, 31), (16, 16, 16))[seed]
    sc = _scene(rng, shape, 2, crowd)
    metal = _numpy_labels(sc, shape)[0] > 0
    a = fractions_from_scene_device(sc, metal, mirror=mirror)
    b = solver3d.fractions_from_scene(sc, metal, mirror=mirror)
    assert np.array_equal(a.view(np.int32), b.view(np.int32))
