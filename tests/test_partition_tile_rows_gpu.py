"""Staged interiors of a partition whose last z tile is more than half full:
the tile rows that were asked for (or chosen with the stages), in every
precision, against the oracle and the bits of the register tiles."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 1e-4}


def _scene(mod, nz, low, high, random):
    nx, ny = 14, 22
    shape = (nx, ny, nz)
    eps = np.random.default_rng(7).uniform(1.0, 3.0, size=shape + (3,)) if random else 2.0
    g = mod.Grid(shape, grid_spacing=100e-9, permittivity=eps)
    g[0:3, :, :] = mod.PML()
    g[:, -3:, :] = mod.PML()
    g[:, :, 0:low] = mod.PML()
    g[:, :, -high:] = mod.PML()
    g[nx // 2, ny // 2, nz // 2] = mod.PointSource(period=12)
    rng = np.random.default_rng(3)
    g.E = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)
    return g


@pytest.mark.parametrize("random", [False, True])
@pytest.mark.parametrize("rows", [0, 4, 8, 16])
@pytest.mark.parametrize("prec,nz,low,high", [("float32", 128, 9, 30), ("float64", 64, 9, 9)])
def test_rows_of_a_staged_interior(fd, prec, nz, low, high, rows, random):
    fd.set_backend("gb300." + prec)
    g = _scene(fd, nz, low, high, random)
    eng = g._ensure_engine()
    eng.set_tuning(pml_mode=4, variant=2, tile_rows=rows)
    t = eng.tiling()
    assert t["pml_split"] == 2 and t["variant"] == 2
    assert t["rows_y"] == rows or rows == 0
    assert t["threads_z"] == (16 if t["rows_y"] == 16 else 32)
    g.run(9, progress_bar=False)
    eng.check_status()
    r = _scene(fd, nz, low, high, random)
    r._ensure_engine().set_tuning(pml_mode=4, variant=1)
    r.run(9, progress_bar=False)
    assert torch.equal(g.E, r.E) and torch.equal(g.H, r.H)
    o = _scene(fo, nz, low, high, random)
    o.run(9)
    assert rel_l2(g.E, o.E) <= TOL[prec] and rel_l2(g.H, o.H) <= TOL[prec]
