"""Absorbing layers registered in other orders than axis by axis: the plan that
small float32 grids get, and the bits of the plan that corrects every layer in
a kernel of its own, in registration order."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo
from test_adjoint_flat_gpu import _gradient

pytestmark = pytest.mark.gpu

# (axis, high, thickness)
INTERLEAVED = {
    "lows_then_highs": [(0, 0, 4), (1, 0, 5), (2, 0, 3), (0, 1, 3), (1, 1, 4), (2, 1, 6)],
    "highs_then_lows": [(2, 1, 6), (1, 1, 4), (0, 1, 3), (0, 0, 4), (2, 0, 3), (1, 0, 5)],
    "z_split_by_y": [(2, 0, 3), (1, 0, 5), (1, 1, 4), (2, 1, 6)],
    "x_split_by_z": [(0, 1, 3), (2, 1, 6), (0, 0, 4)],
}


def _layers(mod, g, spec):
    for axis, high, t in spec:
        if g.shape[axis] == 1:
            continue
        at = [slice(None)] * 3
        at[axis] = slice(-t, None) if high else slice(0, t)
        g[tuple(at)] = mod.PML()


def _scene(mod, shape, spec):
    nx, ny, nz = shape
    eps = np.ones(shape)
    eps[nx // 4:nx // 2, :, nz // 3:] = 4.0
    g = mod.Grid(shape, grid_spacing=155e-9, permittivity=eps)
    _layers(mod, g, spec)
    g[3:nx - 3, 2:ny // 2, :] = mod.Object(permittivity=3.0)
    g[nx // 2, ny // 2, nz // 2] = mod.PointSource(period=11)
    g[:, ny // 2, nz // 2] = mod.LineDetector(name="line")
    rng = np.random.default_rng(3)
    g.E = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)
    g.H = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)
    return g


def _run(fd, shape, spec, steps=12, **tune):
    g = _scene(fd, shape, spec)
    g._ensure_engine().set_tuning(**tune)
    g.run(steps, progress_bar=False)
    g._engine.check_status()
    return g


@pytest.mark.parametrize("shape", [(13, 17, 15), (16, 20, 32), (21, 40, 1)])
@pytest.mark.parametrize("order", sorted(INTERLEAVED))
def test_interleaved_layers(fd, order, shape):
    fd.set_backend("gb300.float32")
    spec = INTERLEAVED[order]
    g = _run(fd, shape, spec)
    assert g._engine.tiling()["persistent"] == 1
    o = _scene(fo, shape, spec)
    o.run(12)
    assert rel_l2(g.E, o.E) <= 1e-4 and rel_l2(g.H, o.H) <= 1e-4
    for tune in (dict(pml_mode=2, variant=1), dict(persistent=1), dict(persistent=2, x_chunk=3)):
        f = _run(fd, shape, spec, **tune)
        assert f._engine.tiling()["persistent"] == (tune.get("persistent") == 2)
        assert torch.equal(f.E, g.E) and torch.equal(f.H, g.H), tune


@pytest.mark.parametrize("order", sorted(INTERLEAVED))
def test_gradient_through_interleaved_layers(fd, order):
    def build(mod):
        g = mod.Grid((12, 17, 18), grid_spacing=155e-9)
        _layers(mod, g, [(a, h, min(t, 4)) for a, h, t in INTERLEAVED[order]])
        obj = mod.Object(permittivity=2.0)
        g[3:6, 4:9, 5:9] = obj
        g[4, 6, 9] = mod.PointSource(period=9)
        g[:, 7, 9] = mod.LineDetector(name="line")
        value = np.random.default_rng(5).uniform(0.3, 0.9, size=(3, 5, 4))
        return g, obj, value, {("line", "E"): np.ones(3), ("line", "H"): np.full(3, 0.5)}, 5

    flat = _gradient(fd, build, "float32", pml_mode=1, variant=1)
    assert np.abs(flat).max() > 0
    assert np.array_equal(flat, _gradient(fd, build, "float32", pml_mode=2, variant=1))
    assert rel_l2(flat, _gradient(fd, build, "float64")) <= 1e-4


# layers that the flat passes do not take
OTHERS = {
    "share_x": [(0, 0, 9), (0, 1, 8), (1, 0, 3), (1, 1, 4)],
    "share_all": [(0, 0, 9), (2, 0, 9), (1, 0, 12), (0, 1, 8), (1, 1, 9), (2, 1, 10)],
}


@pytest.mark.parametrize("shape", [(13, 17, 15), (16, 20, 16), (14, 40, 1)])
@pytest.mark.parametrize("spec", sorted(OTHERS))
def test_layers_of_one_axis_that_share_cells(fd, spec, shape):
    fd.set_backend("gb300.float32")
    spec = OTHERS[spec]
    g = _run(fd, shape, spec)
    assert g._engine.tiling()["persistent"] == 1
    o = _scene(fo, shape, spec)
    o.run(12)
    assert rel_l2(g.E, o.E) <= 1e-4 and rel_l2(g.H, o.H) <= 1e-4
    for tune in (dict(pml_mode=2, variant=1), dict(persistent=1), dict(persistent=2, x_chunk=3)):
        f = _run(fd, shape, spec, **tune)
        assert f._engine.tiling()["persistent"] == (tune.get("persistent") == 2)
        assert torch.equal(f.E, g.E) and torch.equal(f.H, g.H), tune


@pytest.mark.parametrize("prec,shape,split", [
    ("float64", (96, 96, 96), 0), ("float64", (96, 96, 64), 0), ("float64", (128, 128, 64), 2),
    ("float64", (100, 100, 80), 2), ("float32c", (112, 112, 64), 0), ("float32c", (96, 112, 128), 2),
    ("float32c", (104, 104, 104), 2),
])
def test_partition_where_rows_fill_the_tiles(fd, prec, shape, split):
    """Rows that fill the register tiles to the last thread keep mid-sized grids
    in the persistent loop; the partition starts at more cells."""
    fd.set_backend("gb300." + prec)
    g = fd.Grid(shape, grid_spacing=155e-9)
    _layers(fd, g, [(a, h, 10) for a in range(3) for h in range(2)])
    t = g._ensure_engine().tiling()
    assert t["pml_split"] == split and t["persistent"] == (split == 0)


@pytest.mark.parametrize("shape,several,split", [((4000, 4000, 1), True, 1), ((4000, 4000, 1), False, 0),
                                                 ((3500, 3500, 1), True, 0)])
def test_layers_of_large_2d_grids(fd, shape, several, split):
    """The layers of large 2D float32 grids in kernels of their own: where the
    grid runs register tiles (several materials), not flat ones."""
    fd.set_backend("gb300.float32")
    eps = 1.0
    if several:
        eps = np.ones(shape)
        eps[500:900, 300:800] = 4.0
        eps[1500:1700, 800:1100] = 2.25
    g = fd.Grid(shape, grid_spacing=155e-9, permittivity=eps)
    _layers(fd, g, [(0, 0, 16), (0, 1, 16), (1, 0, 16), (1, 1, 16)])
    assert g._ensure_engine().tiling()["pml_split"] == split


@pytest.mark.parametrize("shape,several,staged", [((256, 240, 240), True, True), ((256, 240, 240), False, False),
                                                  ((224, 224, 224), True, False)])
def test_interior_of_a_partition(fd, shape, several, staged):
    """The interior of a float32 partition runs staged where the material is
    indexed (the register tiles read it in full) at fewer cells than where it
    is uniform."""
    fd.set_backend("gb300.float32")
    eps = 1.0
    if several:
        eps = np.ones(shape)
        eps[50:90, 30:80, 20:100] = 4.0
        eps[150:170, 80:110, 60:190] = 2.25
    g = fd.Grid(shape, grid_spacing=155e-9, permittivity=eps)
    _layers(fd, g, [(a, h, 14) for a in range(3) for h in range(2)])
    t = g._ensure_engine().tiling()
    assert t["pml_split"] == 2 and t["variant"] == (2 if staged else 1)
