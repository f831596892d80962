"""Timed work of the framework: what a user's program has it do, through its public entry points.

Three kinds of program use it:

* ``frame``: an interactive or headless frame loop (the reference app's own loop): each frame
  configures, sets the pointer's splats, encodes its substeps call by call (step, dye, CFL
  reduction) and, on every ``diagEvery``-th frame, encodes diagnostics whose readback is
  collected a frame later.
* ``run``: a simulation advanced by a number of graph-replayed steps, then its fields read.
* ``ensemble``: a batch of independent simulations of uneven sizes advanced together, then
  every state and energy read.

A pass advances the simulation by the case's steps and returns the fields a program reads at
that point, whole: the spectral state, the dye texture and the diagnostics.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import __graft_entry__ as entry  # noqa: E402  (loads the package: its folder name is no identifier)

DEV = "cuda"


def _flow(name, kind, n, steps, **kw):
    case = {"name": name, "kind": kind, "n": n, "steps": steps, "dyeScale": 0, "fft": "fp32", "frames": 0,
            "diagEvery": 0, "splats": 0, "beta": 0.0, "drag": 0.01, "viscosity": 1.0, "hyperP": 4,
            "forceAmp": 0.0, "forceK": 0.0, "forceWidth": 1.0, "cfl": 0.5, "dtMin": 1e-6, "dtMax": 1e-3,
            "dyeFade": 0.999, "kmin": 4.0, "kmax": 12.0, "rms": 1.0}
    case.update(kw)
    return case


def listed():
    stir = {"drag": 0.05, "viscosity": 2.0, "hyperP": 2, "dtMax": 0.01, "kmin": 8.0, "kmax": 20.0, "rms": 3.0}
    cascade = {"forceAmp": 0.1, "forceK": 64.0, "forceWidth": 2.0}
    return [
        # the smallest interactive setting: every frame is launches and latency
        _flow("frame_64", "frame", 64, 1, frames=24, dyeScale=2, diagEvery=6, **stir),
        # the app's default grid (256 with a refined dye), two strokes held down, two substeps a frame
        _flow("frame_256_stir", "frame", 256, 2, frames=12, dyeScale=2, diagEvery=6, splats=2, **stir),
        # the 1024 forced cascade frame by frame with diagnostics on every frame (a monitored run)
        _flow("frame_1024_monitor", "frame", 1024, 1, frames=48, dyeScale=2, diagEvery=1, **cascade),
        # free decay at 256 with a passive dye on the same grid, fixed step, Laplacian viscosity
        _flow("decay_256_dye", "run", 256, 200, dyeScale=1, viscosity=7.28, hyperP=1, drag=0.0, dtMin=2e-3,
              dtMax=2e-3, kmin=6.0, kmax=10.0),
        # a 512 beta-plane run without dye, the size of the precision studies
        _flow("beta_512", "run", 512, 300, beta=10.0, viscosity=1.5, hyperP=1, drag=5e-3, dtMax=5e-3, kmin=3.0,
              kmax=9.0),
        # the forced inverse cascade at 1024 with the 2048 dye: the headline workload
        _flow("cascade_1024_dye", "run", 1024, 240, dyeScale=2, **cascade),
        # the same flow alone (spectra and statistics only)
        _flow("cascade_1024", "run", 1024, 300, **cascade),
        # ... and with the tensor-core split transforms
        _flow("cascade_1024_tc", "run", 1024, 120, fft="tc-f16", **cascade),
        # the same cascade one size up
        _flow("cascade_2048", "run", 2048, 100, **cascade),
        # beta-plane jet formation at the largest grid
        _flow("jets_4096", "run", 4096, 60, beta=10.0, drag=5e-3, forceAmp=0.05, forceK=128.0, forceWidth=3.0,
              dtMax=2e-4),
        # parameter studies: 256 simulations at 256, and a mixed batch of uneven grids
        {"name": "ensemble_256", "kind": "ensemble", "n64": 0, "n128": 0, "n256": 256, "n512": 0, "n1024": 0,
         "steps": 120, "dt": 2e-3, "hyperP": 1, "forceAmp": 0.0},
        {"name": "ensemble_mixed", "kind": "ensemble", "n64": 0, "n128": 64, "n256": 128, "n512": 16, "n1024": 0,
         "steps": 150, "dt": 2e-3, "hyperP": 1, "forceAmp": 0.0},
    ]


def draw(rng):
    kind = rng.choice(["frame", "run", "run", "ensemble"])
    if kind == "ensemble":
        case = {"kind": "ensemble", "steps": rng.randint(1, 100), "dt": rng.uniform(5e-4, 2e-3),
                "hyperP": rng.choice([1, 2, 4]), "forceAmp": rng.choice([0.0, 0.0, 0.05])}
        budget = 2 ** rng.uniform(14, 24)          # cells over the batch
        for size in (64, 128, 256, 512, 1024):
            share = rng.random() ** 2 * budget
            case["n%d" % size] = min(int(share / size ** 2), 400)
        if not any(case["n%d" % s] for s in (64, 128, 256, 512, 1024)):
            case["n64"] = rng.randint(1, 9)
        return case
    n = 2 ** rng.randint(5, 12)
    fft = rng.choice(["fp32"] * 5 + ["tc-f16", "tc-bf16"]) if n >= 256 else "fp32"
    dye = rng.choice([0, 1, 2, 2, 4] if n <= 1024 else [0, 0, 1]) if kind == "run" else rng.choice([1, 2, 2])
    if kind == "frame" and n > 2048:
        n = 2048
    weight = n * n * (1.0 + 0.4 * dye * dye) * (4.0 if fft != "fp32" and n != 1024 else 2.0 if fft != "fp32" else 1.0)
    steps_all = max(2, min(300, int(5e8 / weight)))
    kc = n / 3.0
    fk = rng.uniform(0.15, 0.6) * kc
    case = _flow("", kind, n, rng.randint(max(1, steps_all // 3), steps_all), dyeScale=dye, fft=fft,
                 beta=rng.choice([0.0, rng.uniform(0.5, 20.0)]), drag=rng.uniform(0.0, 0.05),
                 viscosity=rng.uniform(0.3, 4.0), hyperP=rng.choice([1, 2, 4]), cfl=0.5,
                 dtMax=rng.choice([2e-4, 1e-3, 5e-3]) if n <= 1024 else rng.choice([1e-4, 2e-4, 1e-3]),
                 kmin=0.1 * kc, kmax=max(4.0, 0.3 * kc), rms=rng.uniform(0.5, 3.0))
    if rng.random() < 0.5:
        case.update(forceAmp=rng.uniform(0.01, 0.1), forceK=fk, forceWidth=rng.uniform(1.0, 4.0))
    if kind == "frame":
        every = rng.choice([1, 3, 6])
        substeps = rng.randint(1, 4)
        ticks = max(1, min(48, steps_all // substeps) // every)
        case.update(steps=substeps, frames=every * ticks, diagEvery=every, splats=rng.choice([0, 0, 1, 3, 8]))
    case.pop("name")
    return case


# ------------------------------------------------------------------ inputs, from the seed alone
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _vorticity(g, n, kmin, kmax, rms, count=1):
    """`count` real random fields with energy between kmin and kmax and the given rms, float32."""
    noise = torch.randn((count, n, n), generator=g, device=DEV, dtype=torch.float32)
    k = torch.fft.fftfreq(n, 1.0 / n, device=DEV)
    kr = torch.sqrt(k[:, None] ** 2 + k[None, :n // 2 + 1].abs() ** 2)
    kept = ((kr >= kmin) & (kr <= kmax)).to(torch.float32)
    w = torch.fft.irfft2(torch.fft.rfft2(noise) * kept, s=(n, n))
    return w * (rms / w.square().mean(dim=(1, 2), keepdim=True).sqrt())


def _dye(g, m):
    """A smooth dye texture: a few random waves per channel, values in [0, 1], alpha 1, binary16."""
    x = (torch.arange(m, device=DEV) + 0.5) * (2 * math.pi / m)
    out = torch.ones((m, m, 4), device=DEV)
    for c in range(3):
        p = torch.rand(4, generator=g, device=DEV) * (2 * math.pi)
        out[..., c] = 0.5 + 0.25 * (torch.sin(3 * x + p[0])[None, :] * torch.sin(2 * x + p[1])[:, None]
                                    + torch.sin((5 * x + p[2])[None, :] + (3 * x + p[3])[:, None]))
    return out.to(torch.float16).cpu().numpy()


def _splats(case, seed):
    """Strokes of the pointer: position, movement, colour, radius, strength and dye amount."""
    r = random.Random(int(seed) * 31 + 5)
    out = []
    for _ in range(case["splats"]):
        dx, dy = r.uniform(-0.006, 0.006), r.uniform(-0.006, 0.006)
        out.append({"x": r.random(), "y": r.random(), "dx": dx, "dy": dy,
                    "color": [r.random(), r.random(), r.random()], "radius": r.uniform(0.02, 0.06), "amp": 400.0,
                    "dyeAmp": min(1.0, math.hypot(dx, dy) * 40)})
    return out


def _flow_inputs(case, seed):
    g = _generator(seed)
    field = _vorticity(g, case["n"], case["kmin"], case["kmax"], case["rms"])[0]
    dye = _dye(g, case["n"] * case["dyeScale"]) if case["dyeScale"] else None
    return field, dye, _splats(case, seed)


SIZES = (64, 128, 256, 512, 1024)


def _members(case, seed):
    """The batch's members: grid size, viscosity, beta, drag, forcing and step of each."""
    r = random.Random(int(seed) * 13 + 3)
    out = []
    for size in SIZES:
        for _ in range(case["n%d" % size]):
            scale = (size / 3.0) ** (2 * case["hyperP"] - 2)
            out.append({"n": size, "beta": r.uniform(0, 20), "drag": r.uniform(0, 2e-2),
                        "nuH": r.uniform(1e-4, 1e-3) / scale, "hyperP": case["hyperP"], "dt": case["dt"],
                        "forceAmp": case["forceAmp"], "forceK": size / 8.0, "forceWidth": 2.0})
    return out


def _member_fields(case, seed):
    """Initial spectra of the members, size by size, complex64 on the GPU: [(n, (count, n, n))]."""
    g = _generator(seed)
    out = []
    for size in SIZES:
        if case["n%d" % size]:
            w = _vorticity(g, size, 4.0, 12.0, 1.0, count=case["n%d" % size])
            out.append((size, torch.fft.fft2(w) * _band(size).to(torch.float32)))
    return out


# ------------------------------------------------------------------ what the program keeps
def _config(case):
    return {k: case[k] for k in ("beta", "drag", "viscosity", "hyperP", "forceAmp", "forceK", "forceWidth", "cfl",
                                 "dtMin", "dtMax", "dyeFade")}


def prepare(case, seed):
    pkg = entry.load_package()
    if case["kind"] == "ensemble":
        ens = pkg.Ensemble(_members(case, seed))
        i = 0
        for _, w in _member_fields(case, seed):
            for spectrum in w.cpu().numpy():
                ens.setState(i, spectrum)
                i += 1
        cells = sum(d["n"] ** 2 for d in ens.instances)
        return {"case": case, "ensemble": ens, "out": np.zeros(cells, np.complex64)}
    field, dye, splats = _flow_inputs(case, seed)
    solver = pkg.Solver.create(n=case["n"], dyeScale=max(1, case["dyeScale"]), fft=case["fft"])
    solver.configure(_config(case))
    solver.reset({"field": field.cpu().numpy(), "dyePattern": "none"})
    if dye is not None:
        solver.setDye(dye.view(np.uint16))
    return {"case": case, "solver": solver, "config": _config(case), "splats": splats}


def _frames(state):
    """The frame loop; returns the diagnostics read last."""
    case, solver = state["case"], state["solver"]
    diag = None
    for tick in range(case["frames"]):
        solver.configure(state["config"])
        solver.setSplats(state["splats"])
        if not solver.primed:
            solver.encodePrime()
        for _ in range(case["steps"]):
            solver.encodeStep()
            solver.encodeDye()
            solver.encodeReduce()
        if (tick + 1) % case["diagEvery"] == 0:
            solver.encodeDiagnostics()
            diag = solver.readDiagnostics() or diag      # the copy of the frame before, if any
            solver.copyDiagnostics()
    return solver.readDiagnostics() or diag


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        ens, out = state["ensemble"], state["out"]
        ens.step(case["steps"])
        at = 0
        for i, d in enumerate(ens.instances):
            cells = d["n"] ** 2
            out[at:at + cells] = ens.getState(i).reshape(-1)
            at += cells
        energy, enstrophy = ens.energy()
        return {"states": out, "energy": energy.astype(np.float32), "enstrophy": enstrophy.astype(np.float32)}
    solver = state["solver"]
    result = {}
    if case["kind"] == "frame":
        d = _frames(state)
        result["spectrum"] = d["spectrum"].astype(np.float32)
        result["zonal"] = d["zonal"]
        result["scalars"] = np.array([d["energy"], d["enstrophy"], d["dt"], d["maxSpeed"]], np.float32)
    else:
        solver.step(case["steps"], dye=case["dyeScale"] > 0, reduce=True, graph=True, relatch=True)
    result["state"] = solver.getBuffer("state%d" % solver.phase)
    if case["dyeScale"]:
        result["dye"] = solver.currentDye.view(np.float16)
    return result


def work(case):
    """Inputs read once, outputs written once; 15 real 2D transforms a step (5 a stage, two of
    them in one complex transform) and the pointwise work of a cell or a dye texel."""
    if case["kind"] == "ensemble":
        cells = [(s, case["n%d" % s] * s * s) for s in SIZES]
        total = sum(c for _, c in cells)
        return {"bytes": 16.0 * total,
                "flops": case["steps"] * sum(c * (75.0 * math.log2(s) + 150.0) for s, c in cells)}
    n, m = case["n"], case["n"] * case["dyeScale"]
    steps = case["steps"] * max(1, case["frames"])
    return {"bytes": 16.0 * n * n + 16.0 * m * m,
            "flops": steps * (n * n * (75.0 * math.log2(n) + 150.0) + 180.0 * m * m)}


# ------------------------------------------------------------------ the same in 64 bits
def _wave(n):
    return torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64)


def _band(n):
    inside = _wave(n).abs() < n / 3.0
    return inside[:, None] & inside[None, :]


class _Flow64:
    """The integrating-factor RK3 step in complex128; `w` may have leading batch dimensions and
    the coefficients matching ones."""

    def __init__(self, n, beta, drag, nu, p):
        k = _wave(n)
        self.n, self.kx, self.ky = n, k[None, :], k[:, None]
        self.k2 = self.kx ** 2 + self.ky ** 2
        self.inv = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), torch.zeros_like(self.k2))
        self.band = _band(n)
        linear = torch.complex(-drag - nu * self.k2 ** p, beta * self.kx * self.inv)
        self.linear = torch.where(self.band, linear, torch.zeros_like(linear))
        self.live = self.band & (self.k2 > 0)

    def fields(self, w):
        u = torch.fft.ifft2(1j * self.ky * self.inv * w).real
        v = torch.fft.ifft2(-1j * self.kx * self.inv * w).real
        return u, v

    def rhs(self, w, force):
        u, v = self.fields(w)
        omega = torch.fft.ifft2(w).real
        f = -(1j * self.kx * torch.fft.fft2(u * omega) + 1j * self.ky * torch.fft.fft2(v * omega))
        return ((f if force is None else f + force) * self.live), u, v

    def step(self, w, dt, force):
        """The state a step later, and the velocity of the last stage's input."""
        half = torch.exp(self.linear * (0.5 * dt))
        full = half * half
        f, _, _ = self.rhs(w, force)
        w1 = full * (w + dt * f)
        f, _, _ = self.rhs(w1, force)
        w2 = 0.75 * half * w + 0.25 * (w1 + dt * f) / half
        f, u, v = self.rhs(w2, force)
        return (full * w + 2.0 * half * (w2 + dt * f)) / 3.0 * self.live, u, v


def _hash(x):
    m = 0xFFFFFFFF
    v = (x * 747796405 + 2891336453) & m
    v = (((v >> ((v >> 28) + 4)) ^ v) * 277803737) & m
    return (v >> 22) ^ v


class _Annulus64:
    """White-in-time forcing of the cells around |k| = forceK, phases hashed from cell and step."""

    def __init__(self, flow, amp, k0, width):
        n = flow.n
        env = torch.exp(-((torch.sqrt(flow.k2) - k0) / width) ** 2)
        rows, cols = torch.nonzero(flow.live & (env > 1e-4), as_tuple=True)
        kx, ky = flow.kx[0, cols], flow.ky[rows, 0]
        first = (ky > 0) | ((ky == 0) & (kx > 0))
        hr, hc = torch.where(first, rows, (n - rows) % n), torch.where(first, cols, (n - cols) % n)
        self.n, self.cell, self.key = n, rows * n + cols, hr * n + hc
        self.sign = torch.where(first, 1.0, -1.0).double()
        self.base = amp * env[rows, cols] * 0.01 * n * n

    def __call__(self, step, dt):
        mixed = self.key ^ int(_hash(int(step)))
        phase = 2.0 * math.pi * _hash(mixed).double() / 4294967296.0
        a = self.base / math.sqrt(max(dt, 1e-6))
        out = torch.zeros(self.n * self.n, dtype=torch.complex128, device=DEV)
        out[self.cell] = torch.complex(a * torch.cos(phase), a * self.sign * torch.sin(phase))
        return out.reshape(self.n, self.n)


def _apart(a, b):
    x = a - b + 0.5
    return x - torch.floor(x) - 0.5


def _centres(n):
    return (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n


def _stir64(flow, splats):
    """Spectrum of the vorticity source of the splats: the curl of Gaussian body forces."""
    n = flow.n
    c = _centres(n)
    total = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    for s in splats:
        rx, ry = _apart(c[None, :], s["x"]), _apart(c[:, None], s["y"])
        r2, sig2 = rx ** 2 + ry ** 2, s["radius"] ** 2
        term = 2.0 * s["amp"] * torch.exp(-r2 / sig2) * (s["dx"] * ry - s["dy"] * rx) / sig2
        total += torch.where(r2 < 9.0 * sig2, term, torch.zeros_like(term))
    return torch.fft.fft2(total) * flow.band


def _corners(tex, px, py):
    """The four texels around normalised positions on a periodic grid, and the weights."""
    m = tex.shape[0]
    gx, gy = px * m - 0.5, py * m - 0.5
    bx, by = torch.floor(gx), torch.floor(gy)
    x0, y0 = bx.long() % m, by.long() % m
    x1, y1 = (x0 + 1) % m, (y0 + 1) % m
    flat = tex.reshape(m * m, -1)
    return [flat[(y * m + x).reshape(-1)].reshape(px.shape + (-1,)) for y, x in
            ((y0, x0), (y0, x1), (y1, x0), (y1, x1))], (gx - bx)[..., None], (gy - by)[..., None]


def _bilinear(tex, px, py):
    (a, b, c, d), fx, fy = _corners(tex, px, py)
    return (a * (1 - fx) + b * fx) * (1 - fy) + (c * (1 - fx) + d * fx) * fy


def _half(x):
    return x.to(torch.float16).double()


def _dye64(dye, u, v, dt, fade, splats):
    """One limited back-and-forth advection of the dye (textures are binary16), then the splats."""
    m = dye.shape[0]
    c = _centres(m)
    px, py = c[None, :].expand(m, m), c[:, None].expand(m, m)
    vel = torch.stack([u, v], dim=-1)

    def trace(h):
        at = _bilinear(vel, px, py) * (0.5 * h)
        at = _bilinear(vel, (px - at[..., 0] + 1) % 1.0, (py - at[..., 1] + 1) % 1.0) * h
        return (px - at[..., 0] + 1) % 1.0, (py - at[..., 1] + 1) % 1.0

    h = dt / (2.0 * math.pi)
    sx, sy = trace(h)
    back = _half(_bilinear(_half(_bilinear(dye, sx, sy)), *trace(-h)))
    around, fx, fy = _corners(dye, sx, sy)
    a = (around[0] * (1 - fx) + around[1] * fx) * (1 - fy) + (around[2] * (1 - fx) + around[3] * fx) * fy
    near = torch.stack(around)
    out = torch.minimum(torch.maximum(1.5 * a - 0.5 * _bilinear(back, sx, sy), near.amin(0)), near.amax(0)) * fade
    for s in splats:
        rx, ry = _apart(px, s["x"]), _apart(py, s["y"])
        r2, sig2 = rx ** 2 + ry ** 2, s["radius"] ** 2
        weight = torch.where(r2 < 9.0 * sig2, s["dyeAmp"] * torch.exp(-r2 / sig2), torch.zeros_like(r2))
        out = out + weight[..., None] * torch.tensor(s["color"], dtype=torch.float64, device=DEV)
    return _half(out)


def _f32(x):
    return float(np.float32(x))


def _exact_flow(case, seed):
    field, dye, splats = _flow_inputs(case, seed)
    n = case["n"]
    splats = [{k: [_f32(c) for c in v] if k == "color" else _f32(v) for k, v in s.items()} for s in splats]
    nu = _f32(case["viscosity"] / (n / 3.0) ** (2 * case["hyperP"]))
    flow = _Flow64(n, _f32(case["beta"]), _f32(case["drag"]), nu, case["hyperP"])
    annulus = None
    if case["forceAmp"] > 0:
        annulus = _Annulus64(flow, _f32(case["forceAmp"]), _f32(case["forceK"]), _f32(case["forceWidth"]))
    stir = _stir64(flow, splats) if splats else None
    w = torch.fft.fft2(field.double()) * flow.live
    dye = None if dye is None else torch.from_numpy(dye[..., :3].copy()).to(DEV).double()
    lo, hi, cfl, fade = (_f32(case[k]) for k in ("dtMin", "dtMax", "cfl", "dyeFade"))

    def limit(u, v):
        speed = float((u.abs() + v.abs()).max())
        return max(min(hi, cfl * (2 * math.pi / n) / speed) if speed > 1e-8 else hi, lo), speed

    dt, speed = limit(*flow.fields(w))
    for i in range(case["steps"] * max(1, case["frames"])):
        # a frame's configure() fixes the forcing's phase for its substeps
        phase = i // case["steps"] * case["steps"] if case["kind"] == "frame" else i
        force = annulus(phase, dt) if annulus else None
        if stir is not None:
            force = stir if force is None else force + stir
        w, u, v = flow.step(w, dt, force)
        if dye is not None:
            dye = _dye64(dye, u, v, dt, fade, splats)
        dt, speed = limit(u, v)
    out = {}
    if case["kind"] == "frame":
        dens = 0.5 * w.abs().square() / float(n) ** 4
        bins = torch.round(torch.sqrt(flow.k2)).long().clamp(max=n // 2)
        spectrum = torch.zeros(n // 2 + 1, dtype=torch.float64, device=DEV)
        spectrum.index_add_(0, bins.reshape(-1), (dens * flow.inv).reshape(-1))
        out["spectrum"] = spectrum
        out["zonal"] = u.mean(dim=1)
        out["scalars"] = torch.tensor([float((dens * flow.inv).sum()), float(dens.sum()), dt, speed],
                                      dtype=torch.float64)
    out["state"] = w
    if dye is not None:
        out["dye"] = torch.cat([dye, torch.ones_like(dye[..., :1])], dim=-1)
    return out


def _exact_ensemble(case, seed):
    members, states, energy, enstrophy = _members(case, seed), [], [], []
    at = 0
    for n, w in _member_fields(case, seed):
        count = w.shape[0]
        mine = members[at:at + count]
        at += count

        def column(key):
            return torch.tensor([_f32(d[key]) for d in mine], dtype=torch.float64, device=DEV)[:, None, None]
        flow = _Flow64(n, column("beta"), column("drag"), column("nuH"), case["hyperP"])
        dt = _f32(case["dt"])
        force = None
        if case["forceAmp"] > 0:
            force = _Annulus64(flow, _f32(case["forceAmp"]), n / 8.0, 2.0)(0, dt)
        w = w.to(torch.complex128)
        for _ in range(case["steps"]):
            w, _, _ = flow.step(w, dt, force)
        dens = 0.5 * w.abs().square() / float(n) ** 4
        states.append(w.reshape(-1))
        energy.append((dens * flow.inv).sum(dim=(1, 2)))
        enstrophy.append(dens.sum(dim=(1, 2)))
    return {"states": torch.cat(states), "energy": torch.cat(energy), "enstrophy": torch.cat(enstrophy)}


def exact(case, seed):
    with torch.no_grad():
        return _exact_ensemble(case, seed) if case["kind"] == "ensemble" else _exact_flow(case, seed)
