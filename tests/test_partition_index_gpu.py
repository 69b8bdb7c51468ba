"""Staged interiors of a partition that read a one-byte material index: their
tensor-map coordinates have to start on 16 bytes in every precision, whatever
the layers' thickness, and their bits are those of the full arrays."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 1e-4, "float32c": 1e-4}


def _scene(mod, thickness):
    nx, ny, nz = shape = (20, 18, 64)
    eps = np.random.default_rng(7).choice([1.0, 1.5, 2.25, 3.0], size=shape)
    g = mod.Grid(shape, grid_spacing=100e-9, permittivity=eps)
    for axis, t in ((0, 3), (1, 3), (2, thickness)):
        for side in (slice(0, t), slice(-t, None)):
            at = [slice(None)] * 3
            at[axis] = side
            g[tuple(at)] = mod.PML()
    g[nx // 2, ny // 2, nz // 2] = mod.PointSource(period=12)
    g[:, :, 40] = mod.PlaneSource(period=18, amplitude=0.5, polarization="x")
    return g


@pytest.mark.parametrize("thickness", [3, 7, 14])
@pytest.mark.parametrize("prec", ["float64", "float32", "float32c"])
def test_indexed_staged_interior(fd, prec, thickness):
    fd.set_backend("gb300." + prec)
    runs = []
    for materials in (0, 1):
        g = _scene(fd, thickness)
        eng = g._ensure_engine()
        eng.set_tuning(pml_mode=4, variant=2, materials=materials)
        t = eng.tiling()
        assert t["pml_split"] == 2 and t["variant"] == 2
        assert (eng.compact_materials()[0] is not None) == (materials == 0)
        g.run(15, progress_bar=False)
        eng.check_status()
        runs.append(g)
    assert torch.equal(runs[0].E, runs[1].E) and torch.equal(runs[0].H, runs[1].H)
    o = _scene(fo, thickness)
    o.run(15)
    assert rel_l2(runs[0].E, o.E) <= TOL[prec] and rel_l2(runs[0].H, o.H) <= TOL[prec]
