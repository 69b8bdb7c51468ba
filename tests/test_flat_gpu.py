"""The flat half steps (float32 grids whose layers run inside the pass): planes
that end inside, on and just past a block, odd and one-cell extents, layers of
unequal thickness, in every order, overlapping and behind a periodic boundary,
more objects and sources than a block keeps at hand, against the CPU oracle;
and the same bits for every x chunk, launch per half step or one per run."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu

TOL32 = 1e-4


def _layers(mod, g, spec):
    for axis, high, t in spec:
        at = [slice(None)] * 3
        at[axis] = slice(-t, None) if high else slice(0, t)
        g[tuple(at)] = mod.PML()


ORDERS = {
    "xyz": [(0, 0, 4), (0, 1, 3), (1, 0, 5), (1, 1, 4), (2, 0, 3), (2, 1, 6)],
    "zxy": [(2, 0, 3), (2, 1, 6), (0, 0, 4), (0, 1, 3), (1, 0, 5), (1, 1, 4)],
    "interleaved": [(0, 0, 4), (1, 0, 5), (2, 0, 3), (2, 1, 6), (0, 1, 3), (1, 1, 4)],
    "yz": [(1, 0, 5), (1, 1, 4), (2, 0, 3), (2, 1, 6)],
    "low_z_only": [(2, 0, 7)],
    "high_y_x": [(1, 1, 1), (0, 1, 2)],
    "overlapping": [(0, 0, 4), (0, 1, 3), (2, 0, 9), (2, 1, 9)],
}


def _scene(mod, shape, order, medium="blocks", periodic="", many=False):
    nx, ny, nz = shape
    eps = np.ones(shape)
    if medium == "blocks":
        eps[nx // 4:nx // 2, :, nz // 3:] = 4.0
    elif medium == "random":
        eps = np.random.default_rng(7).uniform(1, 12, size=shape + (3,))
    g = mod.Grid(shape, grid_spacing=155e-9, permittivity=eps)
    if periodic == "before":
        g[0, :, :] = mod.PeriodicBoundary()
    _layers(mod, g, ORDERS[order])
    if periodic == "after":
        g[:, 0, :] = mod.PeriodicBoundary()
    zs = slice(0, nz) if nz < 6 else slice(2, nz - 2)
    if many:
        for q in range(36):
            x, y = 2 + 2 * (q % 6), 1 + 3 * (q // 6)
            g[x:x + 2, y:y + 3, zs] = mod.Object(permittivity=2.0 + 0.1 * q)
    else:
        g[3:nx - 3, 2:ny // 2, zs] = mod.Object(permittivity=3.0)
        g[nx // 2:nx - 1, ny // 2:ny - 1, zs] = mod.AbsorbingObject(permittivity=2.0, conductivity=2e4)
        g[2:5, ny // 2 - 1:ny // 2 + 3, zs] = mod.AnisotropicObject(permittivity=2.5)
    if many:
        for q in range(6):
            g[4 + q % 3, 5 + q % 2, nz // 2] = mod.PointSource(period=9 + q)
    g[nx // 2, 1:ny - 1, nz // 2] = mod.LineSource(period=11)
    if nz > 6:
        g[:, :, nz // 2 + 1] = mod.PlaneSource(period=17, polarization="x")
    g[:, ny // 2, nz // 2] = mod.LineDetector()
    return g


def _seed(g, shape):
    rng = np.random.default_rng(3)
    g.E = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)
    g.H = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)


CASES = [((13, 17, 15), o, {}) for o in sorted(ORDERS) if o != "overlapping"] + [
    ((11, 13, 14), "overlapping", {}),
    ((9, 16, 16), "xyz", {}),                            # a plane of one block
    ((9, 17, 15), "xyz", dict(medium="random")),       # one cell short of a block
    ((8, 1, 257), "low_z_only", dict(medium="vacuum")),  # one past, a single row
    ((23, 300, 1), "high_y_x", {}),
    ((14, 19, 33), "yz", dict(periodic="before")),
    ((14, 19, 33), "low_z_only", dict(periodic="after")),
    ((16, 20, 21), "zxy", dict(many=True)),
]


@pytest.mark.parametrize("shape,order,more", CASES)
def test_flat_half_steps_against_oracle(fd, shape, order, more):
    if shape[1] == 1:
        more = dict(more)

        def build(mod):
            g = mod.Grid(shape, grid_spacing=155e-9)
            _layers(mod, g, ORDERS[order])
            g[4, 0, 128] = mod.PointSource(period=11)
            return g
    else:
        def build(mod):
            return _scene(mod, shape, order, **more)
    fd.set_backend("gb300.float32")
    o = build(fo)
    _seed(o, shape)
    o.run(12)
    first = None
    for tune in (dict(variant=1, pml_mode=1, persistent=1), dict(variant=1, pml_mode=1, persistent=1, x_chunk=1),
                 dict(variant=1, pml_mode=1, persistent=1, x_chunk=5), dict()):
        g = build(fd)
        _seed(g, shape)
        g._ensure_engine().set_tuning(**tune)
        assert g._engine.tiling()["variant"] == 1
        g.run(12, progress_bar=False)
        g._engine.check_status()
        if first is None:
            first = g
            for a, b in ((g.E, o.E), (g.H, o.H)):
                assert rel_l2(a, b) <= TOL32
        assert torch.equal(g.E, first.E) and torch.equal(g.H, first.H), tune


def test_non_finite_values_stay_where_the_reference_has_them(fd):
    """A difference across the grid's face is dropped whatever the cell holds:
    an infinity beside the face spreads as in the oracle."""
    fd.set_backend("gb300.float32")
    shape = (7, 9, 11)
    pair = []
    for mod in (fd, fo):
        g = mod.Grid(shape, grid_spacing=155e-9)
        _layers(mod, g, [(0, 0, 2), (1, 1, 3), (2, 0, 3)])
        E = np.zeros(shape + (3,))
        for cell in ((0, 4, 5), (6, 4, 5), (3, 0, 5), (3, 8, 5), (3, 4, 0), (3, 4, 10), (2, 5, 3)):
            E[cell] = np.inf
        g.E = E
        with np.errstate(invalid="ignore"):
            if mod is fd:
                g.run(1, progress_bar=False)
            else:
                g.run(1)
        pair.append(g)
    for a, b in ((pair[0].E, pair[1].E), (pair[0].H, pair[1].H)):
        a, b = a.cpu().numpy(), np.asarray(b)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
