"""Soft sources of many points inside the fused passes (one group per source):
lines that fill their bounding box, diagonals found by bisection, points listed
twice, sources that cross in one cell and lines across tile borders, against
the CPU oracle."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu


def _scene(mod, shape):
    nx, ny, nz = shape
    g = mod.Grid(shape, grid_spacing=155e-9)
    g[0:4, :, :] = mod.PML()
    g[-4:, :, :] = mod.PML()
    z = nz // 2
    g[nx // 2, 1:ny - 1, z] = mod.LineSource(period=11, amplitude=0.7)       # fills its box
    g[2:nx - 3, 1:ny - 2, z] = mod.LineSource(period=9)                       # diagonal, crosses the first
    g[[5, 6, 6, 5, 7], [4, 4, 4, 4, 9], [z, z, z, z, z]] = mod.LineSource(period=13)  # points listed twice
    if nz > 1:
        g[3, 5, 1:nz - 1] = mod.LineSource(period=7)
    g[nx // 2, ny // 2, z] = mod.PointSource(period=17)
    g[:, ny // 2, z] = mod.LineDetector(name="detector")
    return g


@pytest.mark.parametrize("prec", ["float64", "float32", "float32c"])
@pytest.mark.parametrize("shape,tune", [((23, 19, 30), {}), ((23, 19, 1), {}), ((17, 300, 1), dict(x_chunk=5)),
                                        ((20, 37, 136), dict(variant=2, pml_mode=2)),
                                        ((20, 37, 136), dict(variant=1, pml_mode=4)),
                                        ((20, 37, 136), dict(variant=1, persistent=1))])
def test_line_sources_against_oracle(fd, prec, shape, tune):
    fd.set_backend("gb300." + prec)
    g, o = _scene(fd, shape), _scene(fo, shape)
    if tune:
        g._ensure_engine().set_tuning(**tune)
    g.run(25, progress_bar=False)
    o.run(25)
    if prec == "float64":
        assert torch.equal(g.E.cpu(), torch.as_tensor(np.asarray(o.E)))
        assert torch.equal(g.H.cpu(), torch.as_tensor(np.asarray(o.H)))
    else:
        assert rel_l2(g.E, o.E) <= 1e-4 and rel_l2(g.H, o.H) <= 1e-4
