"""Workloads of the simulator, as a user's program runs them.

A case names a scene (grid size, precision, absorbing layers, medium, object,
source and detector) and what is done with it: ``run`` advances it with
``grid.run``, ``step`` with a loop of ``grid.step`` calls, and ``adjoint``
differentiates a detector loss with respect to a design region.  Every scene
goes on from fields that fill the whole grid, absorbing layers included, as a
simulation does once its source has been on for a while.

``exact`` restates the time step in plain torch float64 (autograd for the
gradients) and shares only the inputs with the code that is measured.
"""

import math

import numpy as np
import torch

import fdtd_gb300 as fd
from fdtd_gb300 import adjoint

C0 = 299792458.0
ETA0 = 4e-7 * math.pi * C0
SPACING = 155e-9
WAVELENGTH = 1550e-9
DFT_WAVELENGTHS = (1500e-9, 1550e-9, 1600e-9)
CONDUCTIVITY = 1e4


def _case(name, task, precision, shape, pml, steps, medium="vacuum", obj="none", source="point", detector="line",
          layers="xyz", periodic="", checkpoint=0):
    nx, ny, nz = shape
    return {"name": name, "task": task, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "pml": pml,
            "layers": layers, "periodic": periodic, "medium": medium, "object": obj, "source": source,
            "detector": detector, "steps": steps, "checkpoint": checkpoint}


def listed():
    return [
        # the library's first example: a small 2D grid in the default
        # precision, stepped one call at a time (a program that looks at the
        # fields between steps)
        _case("step_2d_161x97_f64", "step", "float64", (161, 97, 1), 10, 10, obj="plain", source="line", layers="xy"),
        # a 2D device layout: most of what this kind of simulator is used for
        _case("run_2d_1500x1100_f32", "run", "float32", (1500, 1100, 1), 16, 100, medium="blocks", source="line",
              layers="xy"),
        # configuration 1: small 3D scene, many steps
        _case("run_64_f32", "run", "float32", (64, 64, 64), 10, 200, obj="plain"),
        # a 3D scene whose size comes from physical dimensions, so no extent
        # is a round number
        _case("run_131x150x97_f32", "run", "float32", (131, 150, 97), 9, 50, medium="blocks", obj="plain",
              source="plane", detector="block"),
        # the same in the compensated precision, for long runs
        _case("run_200x190x150_f32c", "run", "float32c", (200, 190, 150), 12, 25, medium="blocks", obj="absorbing"),
        # configuration 4, forward only: the runs of a design loop's line search
        _case("run_128_f32", "run", "float32", (128, 128, 128), 12, 100, obj="plain", source="plane",
              detector="plane"),
        # configuration 4: one gradient of a design loop
        _case("adjoint_128_f32", "adjoint", "float32", (128, 128, 128), 12, 60, obj="plain", source="plane",
              detector="plane", checkpoint=20),
        # configuration 5 at a quarter of its cells per axis pair: gradient of
        # a spectral loss with respect to permittivity tensors
        _case("adjoint_dft_192x192x96_f32", "adjoint", "float32", (192, 192, 96), 10, 40, obj="anisotropic",
              source="gaussian", detector="dft", checkpoint=20),
        # configuration 2: random medium with a conductive block, both precisions
        _case("run_256_random_f32", "run", "float32", (256, 256, 256), 16, 20, medium="random", obj="absorbing",
              source="plane", detector="block"),
        _case("run_256_random_f64", "run", "float64", (256, 256, 256), 16, 10, medium="random", obj="absorbing",
              source="plane", detector="block"),
        # configuration 5, forward: anisotropic block, spectral detector
        _case("run_384x384x192_aniso_f32", "run", "float32", (384, 384, 192), 20, 20, obj="anisotropic",
              source="gaussian", detector="dft"),
        # configuration 3: the largest grid
        _case("run_768_blocks_f32", "run", "float32", (768, 768, 768), 20, 12, medium="blocks", layers="yz",
              periodic="x"),
    ]


def draw(rng):
    kind = rng.choice(["2d", "small", "small", "middle", "middle", "large", "adjoint"])
    precision = rng.choice(["float32", "float32", "float64", "float32c"])

    def extent(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        # users pick round sizes as often as sizes that follow from a length
        return max(lo, n - n % 8) if rng.random() < 0.4 else n

    def steps(cells, target):
        return max(2, min(200, int(target / cells)))

    if kind == "2d":
        shape = (extent(100, 4000), extent(100, 4000), 1)
        cells = shape[0] * shape[1]
        task = rng.choice(["run", "run", "step"])
        return _drop_name(_case("", task, precision, shape, rng.randint(8, 20),
                                rng.randint(4, 20) if task == "step" else steps(cells, 2e8),
                                medium=rng.choice(["vacuum", "blocks"]), obj=rng.choice(["none", "plain", "absorbing"]),
                                source=rng.choice(["line", "point"]), layers="xy"))
    if kind == "adjoint":
        shape = (extent(48, 200), extent(48, 200), extent(48, 160))
        n = max(8, steps(shape[0] * shape[1] * shape[2], 1e8) // 2)
        aniso = rng.random() < 0.4
        return _drop_name(_case("", "adjoint", rng.choice(["float32", "float32", "float64"]), shape, rng.randint(8, 14),
                                n, obj="anisotropic" if aniso else "plain",
                                source=rng.choice(["plane", "gaussian", "point"]),
                                detector=rng.choice(["dft", "plane"]), checkpoint=max(2, n // 3)))
    lo, hi, target = {"small": (32, 100, 1e8), "middle": (90, 240, 2e8), "large": (240, 448, 5e8)}[kind]
    shape = tuple(extent(lo, hi) for _ in range(3))
    periodic = rng.random() < 0.25
    return _drop_name(_case("", rng.choice(["run", "run", "step"]) if kind == "small" else "run", precision, shape,
                            rng.randint(7, min(20, lo // 4)),
                            steps(shape[0] * shape[1] * shape[2], target),
                            medium=rng.choice(["vacuum", "blocks", "blocks", "random"]),
                            obj=rng.choice(["none", "plain", "absorbing", "anisotropic"]),
                            source=rng.choice(["point", "line", "plane", "gaussian"]),
                            detector=rng.choice(["line", "block", "plane", "dft"]),
                            layers="yz" if periodic else "xyz", periodic="x" if periodic else ""))


def _drop_name(case):
    del case["name"]
    return case


# --- inputs: the same for the measured code and for exact() -----------------------


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _box(n, part):
    """A centred range of n / part cells (the whole axis of a 2D grid's z)."""
    if n == 1:
        return 0, 1
    m = max(2, n // part)
    a = (n - m) // 2
    return a, a + m


def _object_box(case):
    part = 3 if case["task"] == "adjoint" else 4
    return [_box(n, part) for n in _shape(case)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fields(case, rng):
    """E and H, float32: a few standing waves of ten to thirty cells per
    component, of about the amplitude that the source drives."""
    out = []
    for _ in range(2):
        f = torch.empty(_shape(case) + (3,), dtype=torch.float32, device=_device())
        for c in range(3):
            waves = []
            for _ in range(3):
                axes = []
                for n in _shape(case):
                    k, ph = 2 * math.pi / rng.uniform(10.0, 30.0), rng.uniform(0, 2 * math.pi)
                    axes.append(torch.as_tensor(np.cos(k * np.arange(n) + ph), dtype=torch.float32).to(f.device))
                axes[0] = axes[0] * 0.3
                waves.append(axes[0][:, None, None] * axes[1][:, None] * axes[2])
            f[..., c] = waves[0].add_(waves[1]).add_(waves[2])
        out.append(f)
    return out


def _permittivity(case, rng):
    """The grid's permittivity: a number, (nx, ny, nz), or (nx, ny, nz, 3)."""
    shape, dev = _shape(case), _device()
    if case["medium"] == "vacuum":
        return 1.0
    if case["medium"] == "blocks":
        eps = torch.ones(shape, dtype=torch.float64, device=dev)
        values = (1.0, 2.25, 12.1)
        for _ in range(400):
            at = []
            for n in shape:
                m = min(n, max(2, int(rng.uniform(n / 96, n / 12))))
                a = int(rng.integers(0, n - m + 1))
                at.append(slice(a, a + m))
            eps[tuple(at)] = values[int(rng.integers(0, 3))]
        return eps
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 62)))
    eps = torch.rand(shape + (3,), generator=gen, dtype=torch.float64, device=dev) * 11.0 + 1.0
    for axis in range(3):  # 3-cell box filter, edges repeated
        n = shape[axis]
        at = torch.arange(n, device=dev)
        eps = (eps.index_select(axis, (at - 1).clamp(min=0)) + eps
               + eps.index_select(axis, (at + 1).clamp(max=n - 1))) / 3.0
    return eps


def _tensors(shape, rng):
    """Inverse permittivities Q diag(1/lambda) Q^T, lambda in [2, 6], one per cell."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 62)))
    lam = torch.rand(shape + (3,), generator=gen, dtype=torch.float64, device=dev) * 4.0 + 2.0
    q = torch.randn(shape + (4,), generator=gen, dtype=torch.float64, device=dev)
    w, x, y, z = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                       2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                       2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], dim=-1)
    rot = rot.reshape(shape + (3, 3))
    return (rot / lam[..., None, :]) @ rot.transpose(-1, -2)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    got = {"E": None, "H": None, "eps": _permittivity(case, rng)}
    got["E"], got["H"] = _fields(case, rng)
    box = tuple(b - a for a, b in _object_box(case))
    if case["task"] == "adjoint":
        if case["object"] == "anisotropic":
            got["design"] = _tensors(box, rng).to(torch.float32)
        else:
            got["design"] = torch.as_tensor(rng.uniform(1.0 / 12.0, 1.0, size=box), dtype=torch.float32,
                                            device=_device())
        if case["precision"] == "float64":
            got["design"] = got["design"].to(torch.float64)
    elif case["object"] == "anisotropic":
        got["tensors"] = _tensors(box, rng)
    else:
        got["object_eps"] = float(rng.uniform(2.0, 6.0))
    got["amplitude"] = float(rng.uniform(0.5, 1.5))
    return got


def _plane_at(case):
    """z of the source plane and of the detector plane."""
    return case["pml"] + 4, case["nz"] - case["pml"] - 5


def _line_at(case):
    """x of the line source, and its range along y."""
    return case["pml"] + 3, case["ny"] // 4, case["ny"] - case["ny"] // 4


# --- the measured side --------------------------------------------------------------


def prepare(case, seed):
    got = _inputs(case, seed)
    fd.set_backend("gb300." + case["precision"])
    shape, t = _shape(case), case["pml"]
    grid = fd.Grid(shape, grid_spacing=SPACING, permittivity=got.pop("eps"), permeability=1.0)
    for axis, name in enumerate("xyz"):
        if name in case["layers"]:
            for side in (slice(0, t), slice(-t, None)):
                at = [slice(None)] * 3
                at[axis] = side
                grid[tuple(at)] = fd.PML()
    if case["periodic"] == "x":
        grid[0, :, :] = fd.PeriodicBoundary()
    box = tuple(slice(a, b) for a, b in _object_box(case))
    design = None
    if case["task"] == "adjoint":
        design = got["design"].requires_grad_(True)
        grid[box] = (fd.AnisotropicObject if case["object"] == "anisotropic" else fd.Object)(permittivity=3.0,
                                                                                              name="design")
    elif case["object"] == "anisotropic":
        grid[box] = fd.AnisotropicObject(permittivity=3.0, name="tensors")
        grid.tensors.inverse_permittivity = got["tensors"]
    elif case["object"] == "absorbing":
        grid[box] = fd.AbsorbingObject(permittivity=got["object_eps"], conductivity=CONDUCTIVITY)
    elif case["object"] == "plain":
        grid[box] = fd.Object(permittivity=got["object_eps"])
    cx, cy, cz = (n // 2 for n in shape)
    wave = {"period": WAVELENGTH / C0, "amplitude": got["amplitude"]}
    if case["source"] == "point":
        grid[cx, cy, cz] = fd.PointSource(**wave)
    elif case["source"] == "line":
        x, a, b = _line_at(case)
        grid[x, a:b, cz] = fd.LineSource(**wave)
    elif case["source"] == "plane":
        grid[:, :, _plane_at(case)[0]] = fd.PlaneSource(polarization="x", **wave)
    else:
        grid[:, :, _plane_at(case)[0]] = fd.GaussianPlaneSource(polarization="x", **wave)
    if case["detector"] == "line":
        det = fd.LineDetector(name="detector")
        grid[:, cy, cz] = det
    elif case["detector"] == "block":
        det = fd.BlockDetector(name="detector")
        grid[tuple(slice(a, b - 1) for a, b in (_box(n, 8) for n in shape))] = det  # inclusive ranges
    elif case["detector"] == "plane":
        det = fd.PlaneDetector(name="detector")
        grid[:, :, _plane_at(case)[1]] = det
    else:
        det = fd.DFTPlaneDetector(wavelengths=DFT_WAVELENGTHS, name="detector")
        grid[:, :, _plane_at(case)[1]] = det
    grid.E = got["E"]
    grid.H = got["H"]
    return {"grid": grid, "detector": det, "design": design, "task": case["task"], "steps": case["steps"],
            "checkpoint": case["checkpoint"]}


def _loss(out, steps):
    """Transmitted power: per frequency, or over the last third of the run."""
    if "dft" in out:
        return (out["dft"].real ** 2 + out["dft"].imag ** 2).sum()
    return (out["E"][steps - steps // 3:, ..., 2] ** 2).sum()


def run(state):
    grid, det, n = state["grid"], state["detector"], state["steps"]
    if state["task"] == "adjoint":
        p = state["design"]
        p.grad = None
        out = adjoint.run(grid, n, design={grid.design: p}, checkpoint_every=state["checkpoint"])["detector"]
        _loss(out, n).backward()
        return {"E": grid.E, "H": grid.H, "grad": p.grad, "detector": {k: v.detach() for k, v in out.items()}}
    if state["task"] == "step":
        for _ in range(n):
            grid.step()
    else:
        grid.run(n, progress_bar=False)
    if isinstance(det, fd.DFTPlaneDetector):
        return {"E": grid.E, "H": grid.H, "detector": {"dft": det.dft}}
    return {"E": grid.E, "H": grid.H,
            "detector": {"E": det.E.tensor_tail(n), "H": det.H.tensor_tail(n)}}


def work(case):
    """Per time step: E and H read and written once, the materials read once as
    few bits as they hold (nothing where uniform, a byte per cell for blocks of
    a few values, three values per cell for a random medium), the object's
    coefficients read once, the layers' auxiliaries read and written once, the
    records written.  An adjoint pass is one forward and one transposed run;
    what checkpoints cost is the method's own."""
    shape = _shape(case)
    cells = shape[0] * shape[1] * shape[2]
    size = 8 if case["precision"] == "float64" else 4
    value = 2 * size if case["precision"] == "float32c" else size
    box = 1
    for a, b in _object_box(case):
        box *= b - a
    per_object = {"none": 0, "plain": 3, "absorbing": 6, "anisotropic": 9}[case["object"]]
    layer = sum(2 * case["pml"] * (cells // shape["xyz".index(a)]) for a in case["layers"])
    medium = {"vacuum": 0, "blocks": 1, "random": 3 * size}[case["medium"]]
    record = {"line": shape[0], "block": cells // 512, "plane": shape[0] * shape[1],
              "dft": 0}[case["detector"]] * 6 * size
    if case["detector"] == "dft":
        record = shape[0] * shape[1] * 3 * len(DFT_WAVELENGTHS) * 32
    step = 12 * value * cells + medium * cells + per_object * size * box + 8 * size * layer + record
    flops = 30 * cells + 2 * per_object * box + 16 * layer
    passes = 2 if case["task"] == "adjoint" else 1
    return {"bytes": float(step * case["steps"] * passes), "flops": float(flops * case["steps"] * passes)}


# --- exact: the time step in plain torch float64 ------------------------------------


def _slab_profiles(t, high, courant):
    """(bE, cE, bH, cH) along the normal of a layer of t cells."""
    vE = np.arange(0.5, t, 1.0) if high else np.arange(t - 0.5, 0, -1.0)
    vH = np.arange(1.0, t, 1.0) if high else np.arange(t - 1.0, 0, -1.0)
    out = []
    for s in (40 * vE ** 3 / (t + 1) ** 4, np.append(40 * vH ** 3 / (t + 1) ** 4, 0.0)):
        b = np.exp(-(s + 1e-8) * courant)
        out += [torch.as_tensor(b, device=_device()), torch.as_tensor((b - 1.0) * s / (s + 1e-8), device=_device())]
    return out


def _diff(F, c, axis, forward):
    """One-sided difference of component c along an axis, zero on the plane
    that has no neighbour."""
    f = F[..., c]
    n = f.shape[axis]
    d = f.narrow(axis, 1, n - 1) - f.narrow(axis, 0, n - 1)
    zero = torch.zeros_like(f.narrow(axis, 0, 1))
    return torch.cat([d, zero] if forward else [zero, d], dim=axis)


class _Exact:
    def __init__(self, case, got):
        self.case, self.shape = case, _shape(case)
        dims = sum(n > 1 for n in self.shape)
        self.courant = 0.99 * float(dims) ** -0.5
        self.dt = self.courant * SPACING / C0
        self.E, self.H = got["E"].double(), got["H"].double()
        eps = got["eps"]
        if not torch.is_tensor(eps):
            eps = torch.full(self.shape + (1,), eps, dtype=torch.float64, device=_device())
        elif eps.ndim == 3:
            eps = eps[..., None]
        self.inv = 1.0 / eps
        self.box = tuple(slice(a, b) for a, b in _object_box(case))
        self._object(got)
        self.slabs = []
        t = case["pml"]
        for axis, name in enumerate("xyz"):
            if name in case["layers"]:
                for high in (0, 1):
                    shape = list(self.shape)
                    shape[axis] = t
                    psi = [torch.zeros(shape, dtype=torch.float64, device=_device()) for _ in range(4)]
                    self.slabs.append((axis, self.shape[axis] - t if high else 0,
                                       _slab_profiles(t, high, self.courant), psi))
        self.amplitude = got["amplitude"]
        self.period = int(WAVELENGTH / C0 / self.dt + 0.5)

    def _object(self, got):
        kind, box = self.case["object"], self.box
        self.kind, self.coef = kind, None
        if kind == "none":
            return
        if self.case["task"] == "adjoint":
            self.coef = got["design"].double()
            if kind == "plain":
                self.coef = self.coef[..., None].expand(self.coef.shape + (3,))
        elif kind == "anisotropic":
            self.coef = got["tensors"]
        else:
            dims = [s.stop - s.start for s in box]
            ie = torch.full(dims + [3], 1.0 / got["object_eps"], dtype=torch.float64, device=_device())
            # the last plane per component follows the grid's own last plane
            grid = self.inv.expand(self.shape + (3,))
            for c in range(3):
                if dims[c] > 1:
                    at, last = list(box), [slice(None)] * 3
                    at[c], last[c] = -1, -1
                    ie[tuple(last) + (c,)] = grid[tuple(at) + (c,)]
            self.coef = ie
        self.inv = self.inv.clone()
        self.inv[box] = 0.0
        if kind == "absorbing":
            self.f = 0.5 * self.courant * self.coef * CONDUCTIVITY * SPACING * ETA0

    def _value(self, q):
        if self.case["source"] == "gaussian":
            period = WAVELENGTH / C0
            fwhm = 4.0 * period
            sigma = fwhm / (2.0 * math.sqrt(2.0 * math.log(2)))
            t = q * self.dt
            return (self.amplitude * math.exp(-((t - 2.0 * fwhm) ** 2) / (2.0 * sigma ** 2))
                    * math.sin(2 * math.pi * t / period))
        return self.amplitude * math.sin(2 * math.pi * q / self.period)

    def _source(self, F, field, q):
        kind, v = self.case["source"], self._value(q)
        nx, ny, nz = self.shape
        if kind in ("plane", "gaussian"):
            F[:, :, _plane_at(self.case)[0], 0 if field == "E" else 1] = v
        elif field == "H":
            return
        elif kind == "point":
            F[nx // 2, ny // 2, nz // 2, 2] += v
        else:
            x, a, b = _line_at(self.case)
            d = (np.arange(a, b) - (a + (b - a) // 2)) ** 2.0
            profile = np.exp(-(d ** 2) / (2 * (0.5 * d.max()) ** 2))
            F[x, a:b, nz // 2, 2] += torch.as_tensor(profile / profile.sum(), device=F.device) * v

    def _half(self, F, G, field, q):
        """F advanced by the curl of G."""
        sign, forward = (1.0, False) if field == "E" else (-1.0, True)
        scale = sign * self.courant
        D = {(a, c): _diff(G, c, a, forward) for a in range(3) for c in range(3) if a != c}
        curl = [D[1, 2] - D[2, 1], D[2, 0] - D[0, 2], D[0, 1] - D[1, 0]]
        material = self.inv if field == "E" else torch.ones(1, dtype=torch.float64, device=F.device)
        rows = material.expand(material.shape[:-1] + (3,))
        F = torch.stack([F[..., c] + scale * rows[..., c] * curl[c] for c in range(3)], dim=-1)
        if field == "E" and self.coef is not None:
            local = torch.stack([u[self.box] for u in curl], dim=-1)
            if self.kind == "plain":
                F[self.box] = F[self.box] + self.courant * self.coef * local
            elif self.kind == "absorbing":
                F[self.box] = (F[self.box] * ((1 - self.f) / (1 + self.f))
                               + self.courant * self.coef * local / (1 + self.f))
            else:
                F[self.box] = F[self.box] + self.courant * (self.coef @ local[..., None])[..., 0]
        for axis, start, (bE, cE, bH, cH), psi in self.slabs:
            b, c = (bE, cE) if field == "E" else (bH, cH)
            t = b.numel()
            along = [1, 1, 1]
            along[axis] = t
            b, c = b.reshape(along), c.reshape(along)
            gate = torch.ones(t, dtype=torch.float64, device=F.device)
            gate[0 if field == "E" else t - 1] = 0.0  # that difference would leave the layer
            c = c * gate.reshape(along)
            at = tuple(slice(start, start + t) if a == axis else slice(None) for a in range(3))
            m = material[at] if material.ndim > 1 else material
            m = m.expand(m.shape[:-1] + (3,))
            for which, sgn in ((0, -1.0), (1, 1.0)):
                k = which + (0 if field == "E" else 2)
                comp, drive = (axis + 1 + which) % 3, (axis + 2 - which) % 3
                psi[k] = psi[k] * b + D[axis, drive][at] * c
                F[at + (comp,)] = F[at + (comp,)] + scale * sgn * m[..., comp] * psi[k]
        if self.case["periodic"] == "x":
            if field == "E":
                F[0] = F[-1].clone()
            else:
                F[-1] = F[0].clone()
        self._source(F, field, q)
        return F

    def steps(self, n, keep_dft):
        """n steps; the detector's records, or its transform."""
        nx, ny, nz = self.shape
        z = _plane_at(self.case)[1]
        at = {"line": (slice(None), ny // 2, nz // 2), "plane": (slice(None), slice(None), slice(z, z + 1)),
              "dft": (slice(None), slice(None), slice(z, z + 1)),
              "block": tuple(slice(*_box(m, 8)) for m in self.shape)}[self.case["detector"]]
        rec_E, rec_H, dft = [], [], 0.0
        for q in range(n):
            self.E = self._half(self.E, self.H, "E", q)
            if keep_dft:
                e = self.E[at]
                parts = []
                for w in DFT_WAVELENGTHS:
                    theta = 2 * math.pi * (C0 / w) * q * self.dt
                    parts.append(torch.complex(e * math.cos(theta), -e * math.sin(theta)))
                dft = dft + torch.stack(parts)
            else:
                rec_E.append(self.E[at].clone())
            self.H = self._half(self.H, self.E, "H", q)
            if not keep_dft:
                rec_H.append(self.H[at].clone())
        return {"dft": dft} if keep_dft else {"E": torch.stack(rec_E), "H": torch.stack(rec_H)}


def exact(case, seed):
    got = _inputs(case, seed)
    dft = case["detector"] == "dft"
    if case["task"] == "adjoint":
        design = got["design"].double().requires_grad_(True)
        got["design"] = design
        sim = _Exact(case, got)
        del got
        out = sim.steps(case["steps"], dft)
        (grad,) = torch.autograd.grad(_loss(out, case["steps"]), design)
        return {"E": sim.E.detach(), "H": sim.H.detach(), "grad": grad,
                "detector": {k: v.detach() for k, v in out.items()}}
    with torch.no_grad():
        sim = _Exact(case, got)
        del got
        out = sim.steps(case["steps"], dft)
        return {"E": sim.E, "H": sim.H, "detector": out}
