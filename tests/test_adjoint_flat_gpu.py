"""The flat transposed half steps (float32 gradients of grids whose layers run
inside the pass): the float64 gradient to round-off on random scenes (odd and
even extents, 2D, layers on random axes in random order, periodic boundaries
before and after them), and the same bits as the plan that runs the layers in
kernels of their own on planes that end on and just past a block."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from test_adjoint_fuzz_gpu import STEPS, adjoint_scene, loss_of

pytestmark = pytest.mark.gpu


def _gradient(fd, build, precision, **tune):
    fd.set_backend("gb300." + precision)
    g, design, value, weights, k = build(fd)
    g._ensure_engine().set_tuning(**tune)
    p = torch.tensor(value, dtype=torch.float64, device="cuda", requires_grad=True)
    outs = fd.adjoint.run(g, STEPS, design={design: p}, checkpoint_every=k)
    loss_of(outs, weights).backward()
    return p.grad.cpu().numpy()


@pytest.mark.parametrize("seed", range(100, 110))
def test_flat_gradient_of_random_scenes(fd, seed):
    """(Detectors of these scenes may share cells, whose seeds add up in any
    order: round-off, not bits.)"""

    def build(mod):
        return adjoint_scene(mod, seed)[:5]

    flat = _gradient(fd, build, "float32", pml_mode=1, variant=1)
    assert rel_l2(flat, _gradient(fd, build, "float64")) <= 1e-4


@pytest.mark.parametrize("shape", [(9, 16, 16), (7, 15, 17), (10, 257, 1)])
@pytest.mark.parametrize("order", ["xyz", "zyx"])
def test_flat_gradient_at_block_edges(fd, shape, order):
    def build(mod):
        g = mod.Grid(shape, grid_spacing=155e-9, permittivity=np.where(np.arange(shape[0]) < 4, 1.0, 2.25)[:, None, None]
                     * np.ones(shape))
        for axis in order:
            if shape["xyz".index(axis)] == 1:
                continue
            for side in (slice(0, 2), slice(-3, None)):
                at = [slice(None)] * 3
                at["xyz".index(axis)] = side
                g[tuple(at)] = mod.PML()
        zs = slice(0, 1) if shape[2] == 1 else slice(5, 9)
        obj = mod.Object(permittivity=2.0)
        g[3:6, 4:9, zs] = obj
        g[4, 6, shape[2] // 2] = mod.PointSource(period=9)
        g[:, 7, shape[2] // 2] = mod.LineDetector(name="line")
        value = np.random.default_rng(5).uniform(0.3, 0.9, size=(3, 5, zs.stop - zs.start))
        weights = {("line", "E"): np.ones(3), ("line", "H"): np.full(3, 0.5)}
        return g, obj, value, weights, 5

    flat = _gradient(fd, build, "float32", pml_mode=1, variant=1)
    assert np.abs(flat).max() > 0
    assert np.array_equal(flat, _gradient(fd, build, "float32", pml_mode=2, variant=1))
    assert rel_l2(flat, _gradient(fd, build, "float64")) <= 1e-4
