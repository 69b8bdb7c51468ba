"""Objects that share cells on small float32 grids: which passes the plan takes
as they pile up, the oracle's values and the same bits on every route."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu


def _scene(mod, shape, n, seed=True):
    g = mod.Grid(shape, grid_spacing=155e-9)
    g[0:4, :, :] = mod.PML()
    g[-4:, :, :] = mod.PML()
    g[:, 0:3, :] = mod.PML()
    if shape[2] > 1:
        g[:, :, -3:] = mod.PML()
    for q in range(n):
        at = tuple(slice(m // 4 + q, m - m // 4 + q) if m > 1 else slice(0, 1) for m in shape)
        g[at] = (mod.AnisotropicObject(permittivity=2.5), mod.Object(permittivity=2.0),
                 mod.AbsorbingObject(permittivity=1.5, conductivity=2e4))[q % 3]
    g[shape[0] // 2, shape[1] // 2, shape[2] // 2] = mod.PointSource(period=11)
    if seed:
        rng = np.random.default_rng(3)
        g.E = rng.standard_normal(shape + (3,)).astype(np.float32).astype(np.float64)
    return g



@pytest.mark.parametrize("shape,n,persistent,flat", [
    ((64, 64, 64), 3, 1, True), ((128, 128, 128), 1, 1, True), ((128, 128, 128), 2, 0, True),
    ((128, 128, 128), 3, 1, False), ((104, 167, 145), 1, 0, True), ((400, 400, 1), 3, 1, True),
    ((900, 900, 1), 1, 1, True), ((900, 900, 1), 2, 1, False),
])
def test_routes(fd, shape, n, persistent, flat):
    fd.set_backend("gb300.float32")
    g = _scene(fd, shape, n, seed=False)
    t = g._ensure_engine().tiling()
    assert (t["persistent"], t["threads_z"] == 256) == (persistent, flat)
    g._engine.set_tuning(persistent=2)
    assert g._engine.tiling()["persistent"] == 1


@pytest.mark.parametrize("shape", [(60, 40, 45), (60, 40, 44), (70, 400, 1)])
@pytest.mark.parametrize("n", [1, 2, 3, 6])
def test_stacks_against_oracle(fd, shape, n):
    fd.set_backend("gb300.float32")
    o = _scene(fo, shape, n)
    o.run(8)
    first = None
    for tune in (dict(), dict(persistent=1), dict(persistent=2), dict(pml_mode=2, variant=1)):
        g = _scene(fd, shape, n)
        g._ensure_engine().set_tuning(**tune)
        g.run(8, progress_bar=False)
        g._engine.check_status()
        assert rel_l2(g.E, o.E) <= 1e-4 and rel_l2(g.H, o.H) <= 1e-4, tune
        first = first or g
        assert torch.equal(g.E, first.E) and torch.equal(g.H, first.H), tune
