"""How the flat, register-streaming and shell kernels read the materials (one
triple, an index, the full arrays), and that they follow changes of the
material arrays in place: against the CPU oracle."""

import numpy as np
import pytest
import torch

from helpers import rel_l2
from oracle import fdtd_oracle as fo

pytestmark = pytest.mark.gpu

TOL = {"float64": 1e-12, "float32": 1e-4, "float32c": 1e-4}


def _scene(mod, shape, medium):
    nx, ny, nz = shape
    rng = np.random.default_rng(7)
    eps = {"uniform": 2.0, "levels": rng.choice([1.0, 1.5, 2.25, 3.0], size=shape),
           "random": rng.uniform(1.0, 3.0, size=shape + (3,))}[medium]
    g = mod.Grid(shape, grid_spacing=100e-9, permittivity=eps, permeability=1.0)
    for axis in range(3):
        if shape[axis] == 1:
            continue
        for side in (slice(0, 3), slice(-3, None)):
            at = [slice(None)] * 3
            at[axis] = side
            g[tuple(at)] = mod.PML()
    g[nx // 2, ny // 2, nz // 2] = mod.PointSource(period=12)
    g[2:nx - 2, ny // 2, nz // 2] = mod.LineDetector(name="line")
    return g


UNIFORM = ("uniform", 1)  # (an index's table lists every combination of the components' four values)


@pytest.mark.parametrize("prec,shape,medium,tune,modes", [
    ("float32", (20, 18, 32), "uniform", {}, [UNIFORM, UNIFORM]),
    ("float32", (20, 18, 30), "levels", {}, [None, UNIFORM]),
    ("float32", (20, 18, 32), "levels", {}, [("index", 64), UNIFORM]),
    ("float32", (20, 18, 32), "random", {}, [None, UNIFORM]),
    ("float32", (20, 18, 32), "levels", dict(materials=1), [None, None]),
    ("float32", (20, 18, 32), "levels", dict(pml_mode=4, variant=1), [None, UNIFORM]),
    ("float32", (20, 18, 32), "levels", dict(pml_mode=4, variant=2), [("index", 64), UNIFORM]),
    ("float32", (20, 18, 32), "levels", dict(step_fusion=2), [("index", 64), UNIFORM]),
    ("float64", (20, 18, 32), "uniform", {}, [None, UNIFORM]),
    ("float64", (20, 18, 32), "uniform", dict(persistent=1), [UNIFORM, UNIFORM]),
    ("float32c", (20, 18, 32), "levels", dict(persistent=1), [None, UNIFORM]),
])
def test_reported_modes(fd, prec, shape, medium, tune, modes):
    fd.set_backend("gb300." + prec)
    g = _scene(fd, shape, medium)
    eng = g._ensure_engine()
    eng.set_tuning(**tune)
    assert eng.compact_materials() == modes


PLANS = [dict(), dict(persistent=1), dict(pml_mode=2, variant=1), dict(pml_mode=4, variant=1), dict(pml_mode=4, variant=2)]


@pytest.mark.parametrize("plan", range(len(PLANS)))
@pytest.mark.parametrize("medium", ["uniform", "levels"])
@pytest.mark.parametrize("prec", ["float32", "float32c", "float64"])
def test_in_place_changes_are_followed(fd, prec, medium, plan):
    fd.set_backend("gb300." + prec)
    shape = (20, 18, 32)
    g, o = _scene(fd, shape, medium), _scene(fo, shape, medium)
    eng = g._ensure_engine()
    eng.set_tuning(**PLANS[plan])

    def step(n):
        g.run(n, progress_bar=False)
        o.run(n)
        assert rel_l2(g.E, o.E) <= TOL[prec] and rel_l2(g.H, o.H) <= TOL[prec]

    step(6)
    for a in (g, o):  # the same layout: another uniform value, or one of the levels
        if medium == "uniform":
            a.inverse_permittivity[...] = 0.4
        else:
            a.inverse_permittivity[8:12, 7:11, 12:20] = 1.0 / 1.5
    step(6)
    for a in (g, o):  # new values
        a.inverse_permittivity[9:12, 8:10, 12:17] = 0.3
        a.inverse_permeability[7:9, 6:12, 14:18] = 0.5
    g.step()
    o.step()
    step(6)
    # a write that torch does not count, and the array assigned to itself
    g.inverse_permittivity.data[6:9, 5:12, 11:20] = 0.7
    g.inverse_permittivity = g.inverse_permittivity
    o.inverse_permittivity[6:9, 5:12, 11:20] = 0.7
    step(6)
