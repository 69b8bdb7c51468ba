"""The interior/shell partition as mid-sized grids get it, on rows that divide
into vectors, into pairs and into nothing: against the CPU oracle, with
objects and sources across the interior's faces and a periodic boundary, and
float32 gradients against the fused plan's."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu

TOL32 = 1e-4


def _scene(mod, shape, periodic=False, order="xyz"):
    nx, ny, nz = shape
    eps = np.ones(shape)
    eps[nx // 4:nx // 2, :, nz // 3:] = 4.0
    g = mod.Grid(shape, grid_spacing=155e-9, permittivity=eps)
    for axis in order:
        if periodic and axis == "x":
            continue
        for side in (slice(0, 9), slice(-8, None)):
            at = [slice(None)] * 3
            at["xyz".index(axis)] = side
            g[tuple(at)] = mod.PML()
    if periodic:
        g[0, :, :] = mod.PeriodicBoundary()
    design = mod.Object(permittivity=3.0, name="design")
    g[4:nx // 3, 6:ny // 2, 5:nz // 2] = design
    g[nx // 2:nx - 3, ny // 2 + 1:ny - 2, 3:nz - 4] = mod.AbsorbingObject(permittivity=2.0, conductivity=2e4)
    g[nx // 2, 3:ny - 3, nz // 2] = mod.LineSource(period=11)
    g[:, :, 10] = mod.PlaneSource(period=17, polarization="x")
    g[:, ny // 2, nz // 2] = mod.LineDetector(name="line")
    return g


def _seed(g, shape, scale=1.0):
    rng = np.random.default_rng(3)
    g.E = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64) * scale
    g.H = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64) * scale


SHAPES = {"float64": [(83, 82, 84), (83, 82, 87), (83, 82, 90)], "float32c": [(95, 94, 96), (95, 94, 99), (95, 94, 98)],
          "float32": [(172, 171, 172), (172, 171, 175), (172, 171, 174)]}


@pytest.mark.parametrize("which", range(3))
@pytest.mark.parametrize("prec,periodic,order", [("float64", False, "xyz"), ("float64", True, "zxy"),
                                                 ("float32c", False, "zxy"), ("float32", False, "xyz")])
def test_automatic_partition_against_oracle(fd, prec, periodic, order, which):
    shape = SHAPES[prec][which]
    fd.set_backend("gb300." + prec)
    g, o = _scene(fd, shape, periodic, order), _scene(fo, shape, periodic, order)
    _seed(g, shape)
    _seed(o, shape)
    assert g._ensure_engine().tiling()["pml_split"] == 2
    steps = 6
    g.run(steps, progress_bar=False)
    o.run(steps)
    if prec == "float64":
        assert torch.equal(g.E.cpu(), torch.as_tensor(np.asarray(o.E)))
        assert torch.equal(g.H.cpu(), torch.as_tensor(np.asarray(o.H)))
    else:
        assert rel_l2(g.E, o.E) <= 1e-4 and rel_l2(g.H, o.H) <= 1e-4


@pytest.mark.parametrize("prec", ["float64", "float32"])
@pytest.mark.parametrize("which", range(3))
def test_gradient_of_automatic_partition_equals_fused(fd, prec, which):
    shape = SHAPES[prec][which]
    fd.set_backend("gb300." + prec)
    grads = []
    for mode in (0, 1):
        g = fd.Grid(shape, grid_spacing=155e-9)
        for axis in range(3):
            for side in (slice(0, 9), slice(-8, None)):
                at = [slice(None)] * 3
                at[axis] = side
                g[tuple(at)] = fd.PML()
        obj = fd.Object(permittivity=2.0)
        g[5:20, 30:41, 7:30] = obj
        g[12, 35, 20] = fd.PointSource(period=9)
        g[:, 33, 18] = fd.LineDetector(name="line")
        g._ensure_engine().set_tuning(pml_mode=mode, variant=mode)
        assert g._engine.tiling()["pml_split"] == (2 if mode == 0 else 0)
        p = torch.tensor(np.random.default_rng(1).uniform(0.3, 0.9, size=(15, 11, 23)), device="cuda",
                         requires_grad=True)
        out = fd.adjoint.run(g, 14, design={obj: p}, checkpoint_every=5)["line"]
        ((out["E"].double() ** 2).sum() + (out["H"].double() ** 2).sum()).backward()
        grads.append(p.grad.cpu().numpy())
    assert np.abs(grads[0]).max() > 0
    assert np.array_equal(grads[0], grads[1])


@pytest.mark.parametrize("shape,obj", [((1201, 1003, 1), True), ((1251, 2003, 1), False)])
def test_large_2d_grids_of_several_materials(fd, shape, obj):
    """Such grids take register tiles of one cell per thread, call by call and
    in the persistent loop."""
    def build(mod):
        eps = np.ones(shape)
        eps[200:500, :] = 4.0
        g = mod.Grid(shape, grid_spacing=155e-9, permittivity=eps)
        g[0:8, :, :] = mod.PML()
        g[-8:, :, :] = mod.PML()
        g[:, 0:9, :] = mod.PML()
        g[:, -9:, :] = mod.PML()
        if obj:
            g[600:900, 300:700, 0] = mod.AbsorbingObject(permittivity=2.0, conductivity=2e4)
        g[550, 20:980, 0] = mod.LineSource(period=11)
        g[:, 500, 0] = mod.LineDetector()
        return g

    fd.set_backend("gb300.float32")
    rng = np.random.default_rng(3)
    E, H = (rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64) for _ in range(2))
    o = build(fo)
    o.E, o.H = E.copy(), H.copy()
    o.run(5)
    first = None
    for persistent in (1, 2, 0):
        g = build(fd)
        g.E, g.H = E, H
        g._ensure_engine().set_tuning(persistent=persistent)
        assert g._engine.tiling()["variant"] == 1
        g.run(5, progress_bar=False)
        g._engine.check_status()
        if first is None:
            first = g
            for a, b in ((g.E, o.E), (g.H, o.H)):
                assert rel_l2(a, b) <= TOL32
        assert torch.equal(g.E, first.E) and torch.equal(g.H, first.H), persistent
