"""The persistent loop over more flat tiles than the GPU holds blocks (thin
grids of large planes): tiles drawn by ticket, their columns worked out per
tile, against the bits of one launch per half step."""

import numpy as np
import pytest
import torch

from test_adjoint_flat_gpu import _gradient

pytestmark = pytest.mark.gpu

SHAPE = (6, 401, 311)  # 488 chunks of a plane


def _grid(mod):
    nx, ny, nz = SHAPE
    eps = np.ones(SHAPE)
    eps[:, 100:180, 50:200] = 4.0
    g = mod.Grid(SHAPE, grid_spacing=155e-9, permittivity=eps)
    g[:, 0:7, :] = mod.PML()
    g[:, -5:, :] = mod.PML()
    g[:, :, 0:6] = mod.PML()
    g[:, :, -9:] = mod.PML()
    return g


def _scene(mod, sources):
    g = _grid(mod)
    g[1:5, 190:260, 100:211] = mod.Object(permittivity=2.0)
    for q in range(sources):
        g[1 + q % 4, 40 + 60 * q, 30 + 50 * q] = mod.PointSource(period=9 + q)
    g[3, 5:390, 4:300] = mod.LineSource(period=13)
    g[2, 200, :] = mod.LineDetector(name="line")
    rng = np.random.default_rng(3)
    g.E = rng.standard_normal(SHAPE + (3,)).astype(np.float32)
    g.H = rng.standard_normal(SHAPE + (3,)).astype(np.float32)
    return g


@pytest.mark.parametrize("sources", [1, 5])
def test_more_tiles_than_blocks(fd, sources):
    fd.set_backend("gb300.float32")
    runs = []
    for persistent in (1, 2):
        g = _scene(fd, sources)
        g._ensure_engine().set_tuning(persistent=persistent, pml_mode=1)
        assert g._engine.tiling()["persistent"] == (persistent == 2)
        g.run(9, progress_bar=False)
        g.run(4, progress_bar=False)
        g._engine.check_status()
        runs.append(g)
    assert torch.equal(runs[0].E, runs[1].E) and torch.equal(runs[0].H, runs[1].H)
    assert torch.equal(runs[0].line.E.tensor(), runs[1].line.E.tensor())
    assert float(runs[0].E.abs().max()) > 0


def test_more_tiles_than_blocks_with_captured_curls(fd):
    def build(mod):
        g = _grid(mod)
        obj = mod.Object(permittivity=2.0)
        g[2:5, 190:240, 100:171] = obj
        g[3, 200, 120] = mod.PointSource(period=9)
        g[3, 202, :] = mod.LineDetector(name="line")
        value = np.random.default_rng(5).uniform(0.3, 0.9, size=(3, 50, 71))
        return g, obj, value, {("line", "E"): np.ones(3), ("line", "H"): np.full(3, 0.5)}, 6

    a = _gradient(fd, build, "float32", persistent=1, pml_mode=1)
    b = _gradient(fd, build, "float32", persistent=2, pml_mode=1)
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
