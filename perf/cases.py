"""Workloads of the fire framework as its users run them, for timing and for checking results.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  the simulation, solver or renderer a program holds before the call, with its inputs
  run(state)           one pass through the public entry points; returns the results
  work(case)           the bytes and operations one pass cannot do without
  exact(case, seed)    what run returns, in 64-bit arithmetic (plain torch), where that has a value

A simulation starts in a burning state: plumes over the seeded spots with smooth random velocities, written
straight into the simulation's fields (its zero-copy views), so every pass advances a fire as a program's frame
loop does.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path.cwd() / "procedural-fire_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import fire_sim as F  # noqa: E402

DEV = "cuda:0"


# ------------------------------------------------------------------------------------------------ the cases
def _step(name, res, cell, dt, emitter, spots, cycles, tol=0.0, omega=1.0):
    """tol = 0: `cycles` V-cycles every step; tol > 0: V-cycles to that relative residual, `cycles` at most."""
    return {"name": name, "kind": "step", "nx": res[0], "ny": res[1], "nz": res[2], "cell": cell, "dt": dt,
            "emitter": emitter, "spots": spots, "cycles": cycles, "tol": tol, "omega": omega}


def listed():
    return [
        # a preview fire or one of many small agents' fires: the smallest grid of the ensemble workload, where
        # launches and the coarse levels' latency are the whole step
        _step("step-32x64x32", (32, 64, 32), 0.0125, 1 / 120, "spots", 3, 4),
        # a grid fitted to a scene instead of to the solver: partial tiles, a hierarchy that stops at odd sizes
        _step("step-50x98x50", (50, 98, 50), 0.0125, 1 / 120, "spots", 4, 3),
        # FireSim's defaults: the page's campfire with logs and coal bed, two cycles a step
        _step("step-80x120x80-campfire", (80, 120, 80), 0.015, 1 / 120, "campfire", 0, 2),
        # the throughput workload: full physics, pressure to 1e-5 with over-relaxed smoothing
        _step("step-128x256x128-tol", (128, 256, 128), 0.005, 1 / 240, "spots", 6, 8, 1e-5, 1.2),
        # an offline simulation: every field far larger than the L2
        _step("step-256x512x256", (256, 512, 256), 0.0025, 1 / 480, "spots", 8, 4),
        # many independent fires of uneven sizes, one batched step for all (data generation)
        {"name": "ensemble-16", "kind": "ensemble", "per_grid": 4, "scale": 1.0, "cycles": 4},
        # one iteration of a source fit: rollout from a stored state, loss, spot-flux gradients
        {"name": "fit-64x128x64", "kind": "fit", "nx": 64, "ny": 128, "nz": 64, "steps": 10, "every": 5, "spots": 8},
        # the pressure solver on its own: a small FP32 solve, half-precision storage at the step's size, and
        # FP32-storage refinement at the size of the solver's own benchmark
        {"name": "poisson-64-fp32", "kind": "poisson", "nx": 64, "ny": 64, "nz": 64, "form": "fp32", "tol": 1e-4},
        {"name": "poisson-128x256x128-fp16", "kind": "poisson", "nx": 128, "ny": 256, "nz": 128, "form": "fp16", "tol": 1e-6},
        {"name": "poisson-256x512x256-ir32", "kind": "poisson", "nx": 256, "ny": 512, "nz": 256, "form": "ir32", "tol": 1e-6},
        # one frame of the renderer's fire passes at the capture size with its default volume scale, and the
        # image read back (the only way out of a headless render)
        {"name": "render-540x960", "kind": "render", "nx": 80, "ny": 120, "nz": 80, "width": 1080, "height": 1920, "scale": 0.5,
         "cubic": 0, "sharp": 0.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, lo, hi, step=1):
    """A grid about twice as tall as wide, its sides multiples of `step`."""
    n = _log(rng, lo, hi)
    r = lambda v: max(step * 2, int(round(v / step)) * step)
    return r(n), r(n * rng.uniform(1.4, 2.1)), r(n * rng.uniform(0.8, 1.1))


def draw(rng):
    kind = rng.choice(["step", "step", "tol", "campfire", "ensemble", "fit", "poisson", "poisson", "render"])
    if kind in ("step", "tol", "campfire"):
        res = _grid(rng, 26, 190, rng.choice([1, 2, 8, 16]))
        cell = 0.64 / res[0]
        tol = 1e-4 if kind == "tol" else 0.0
        c = _step("", res, cell, 1 / rng.choice([60, 120, 240]), "campfire" if kind == "campfire" else "spots", rng.randint(1, 8),
                  8 if tol else rng.randint(1, 4), tol, 1.2 if tol else 1.0)
        del c["name"]
        return c
    if kind == "ensemble":
        return {"kind": "ensemble", "per_grid": rng.randint(1, 4), "scale": rng.choice([0.5, 0.75, 1.0]), "cycles": rng.randint(1, 4)}
    if kind == "fit":
        nx, ny, nz = _grid(rng, 24, 60, rng.choice([2, 8]))
        n = rng.randint(4, 10)
        return {"kind": "fit", "nx": nx, "ny": ny, "nz": nz, "steps": n, "every": rng.randint(2, n), "spots": rng.randint(1, 8)}
    if kind == "poisson":
        nx, ny, nz = _grid(rng, 24, 200, rng.choice([1, 2, 8, 16]))
        form = rng.choice(["fp32", "ir32", "fp16", "bf16"])
        return {"kind": "poisson", "nx": nx, "ny": ny, "nz": nz, "form": form, "tol": 1e-4 if form == "fp32" else 1e-6}
    nx, ny, nz = _grid(rng, 32, 128, rng.choice([1, 2, 8]))
    cubic = rng.choice([0, 0, 1])
    return {"kind": "render", "nx": nx, "ny": ny, "nz": nz, "width": rng.randint(320, 1080), "height": rng.randint(480, 1400),
            "scale": rng.choice([0.5, 0.75]), "cubic": cubic, "sharp": 0.6 if cubic else 0.0}


def _fixed(case):
    return case["tol"] == 0.0


# ------------------------------------------------------------------------------------------------ inputs
class _View:
    """A simulation field's device memory (fire_sim_field) for torch; keeps the simulation alive."""

    def __init__(self, sim, name):
        d = sim.field(name)
        shape = (d.dims[2], d.dims[1], d.dims[0]) + ((d.channels,) if d.channels > 1 else ())
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4" if d.elem_bytes == 4 else "<f2", "data": (d.data, False),
                                         "version": 2}


def _view(sim, name):
    return torch.as_tensor(_View(sim, name), device=DEV)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _smooth(res, channels, gen, cells=6):
    """Band-limited noise in about [-1, 1]: white noise every `cells` cells, trilinear between."""
    nx, ny, nz = res
    low = torch.randn((1, channels, max(2, nz // cells), max(2, ny // cells), max(2, nx // cells)), generator=gen, device=DEV)
    f = torch.nn.functional.interpolate(low, size=(nz, ny, nx), mode="trilinear", align_corners=False)[0]
    return f.mul_(0.6).permute(1, 2, 3, 0)


def _burning(sim, spots, gen):
    """Writes a burning state into vel, S and S2: a hot, rising, sooting plume over every spot, ambient air elsewhere."""
    nx, ny, nz = sim.res
    ax = [torch.arange(n, device=DEV, dtype=torch.float32).add_(0.5).mul_(sim.dx) for n in (nx, ny, nz)]
    x, y, z = ax[0].view(1, 1, nx) + sim.origin[0], ax[1].view(1, ny, 1), ax[2].view(nz, 1, 1) + sim.origin[2]
    top = 0.45 * ny * sim.dx
    plume = torch.zeros((nz, ny, nx), device=DEV)
    for sx, _, sz, sigma, flux in spots.tolist():
        w = 1.3 * sigma + 0.12 * y
        plume += (0.5 + flux / 8) * torch.exp(-((x - sx) ** 2 + (z - sz) ** 2) / (2 * w * w)) * torch.exp(-((y / top) ** 2))
    n = _smooth(sim.res, 4, gen)
    plume = (plume * (1 + 0.5 * n[..., 3])).clamp_(0, 1.15)
    rise = plume.clamp(max=1)
    vel, S, S2 = _view(sim, "vel"), _view(sim, "S"), _view(sim, "S2")
    vel[..., 0] = (0.03 + 0.6 * rise) * n[..., 0]
    vel[..., 1] = 2.2 * rise * (0.25 + y / top).clamp(max=1) + (0.03 + 0.5 * rise) * n[..., 1]
    vel[..., 2] = (0.03 + 0.6 * rise) * n[..., 2]
    vel[..., 3] = 0
    hot = (plume - 0.05).clamp_(min=0)
    S[..., 0] = 1.2 * hot
    S[..., 1] = 0.12 * rise * torch.exp(-y / (0.3 * top))
    S[..., 2] = (2.0 * hot * (y / top).clamp(max=1)).clamp_(max=2.5)
    S[..., 3] = 0.8 * hot * torch.exp(-y / (0.4 * top))
    S2[..., 0] = 0.8 * rise * (0.1 + y / top).clamp(max=1)
    S2[..., 1] = 0.05 * rise
    S2[..., 2] = 0.02 * rise * (y / top)
    S2[..., 3] = 0.3 * rise


def _spots(n, seed, width):
    return F.make_spots(int(seed) % 100000 + 1, n, 1.0, 4.0, 0.02 * width / 0.64, 0.3 * width)


def _sim(case, seed, logs=None, **solver):
    res = (case["nx"], case["ny"], case["nz"])
    sim = F.FireSim(res=res, size=tuple(case["cell"] * n for n in res), logs=logs, **solver)
    spots = _spots(max(case["spots"], 3), seed, res[0] * case["cell"])
    if logs is None:
        sim.set_spots(spots[:case["spots"]])
        sim.set_bed_gain(0.0)
        sim.set_params({"vortEps": 0.3, "turbAmp": 0.2})
        sim.set_soot_age(0.02, 0.06)
    sim.set_params({"seed": float(int(seed) % 1000)})
    _burning(sim, spots, _generator(seed))
    return sim


def _ensemble_grids(case):
    s = case["scale"]
    return [tuple(int(v * s) for v in g) for g in ((32, 64, 32), (48, 96, 48), (64, 128, 64), (96, 192, 96)) for _ in range(case["per_grid"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        logs = F.build_campfire(7) if case["emitter"] == "campfire" else None
        fixed = _fixed(case)
        sim = _sim(case, seed, logs, vcycles=case["cycles"] if fixed else 4, mg_max_cycles=0 if fixed else case["cycles"], mg_tol=case["tol"])
        if case["omega"] != 1.0:
            sim.set_mg_omega(case["omega"])
        return {"kind": kind, "sim": sim, "dt": case["dt"], "out": {n: _view(sim, n) for n in ("vel", "S", "S2", "p")}}
    if kind == "ensemble":
        cell = 0.0125 / case["scale"]
        grids = _ensemble_grids(case)
        ens = F.Ensemble([{"res": g, "size": tuple(cell * v for v in g)} for g in grids], vcycles=case["cycles"])
        for i, (s, g) in enumerate(zip(ens.members, grids)):
            spots = _spots(2 + (i * 5 + int(seed)) % 7, seed + 31 * i, g[0] * cell)
            s.set_spots(spots)
            s.set_params({"seed": float(1000 + i), "vortEps": 0.3, "turbAmp": 0.2})
            s.set_soot_age(0.02, 0.06)
            s.set_bed_gain(0.0)
            s.ensemble = ens
            _burning(s, spots, _generator(seed + 7919 * i))
        return {"kind": kind, "ens": ens, "dt": 1 / 120, "out": [{n: _view(s, n) for n in ("vel", "S", "S2")} for s in ens.members]}
    if kind == "fit":
        sim = _sim(dict(case, cell=0.64 / case["nx"]), seed, mg_max_cycles=8, mg_tol=1e-5)
        sim.set_mg_omega(1.2)
        views = {n: _view(sim, n) for n in ("vel", "S", "S2", "p")}
        start = {n: v.clone() for n, v in views.items()}
        noise = _smooth(sim.res, 4, _generator(seed + 5))
        target = (start["S"] * (1 + 0.1 * noise)).cpu().numpy()
        return {"kind": kind, "sim": sim, "adj": F.Adjoint(sim, case["steps"], case["every"]), "views": views, "start": start,
                "target": target, "spots": case["spots"]}
    if kind == "poisson":
        res = (case["nx"], case["ny"], case["nz"])
        gen = _generator(seed)
        b = torch.zeros(res[::-1], device=DEV)
        c = [torch.arange(n, device=DEV, dtype=torch.float32) + 0.5 for n in res]
        for u in torch.rand((32, 5), generator=gen, device=DEV).tolist():   # Gaussian sources, sigma 1-4 cells
            s = 1 + 3 * u[3]
            g = [torch.exp(-((a - u[i] * n) ** 2) / (2 * s * s)) for i, (a, n) in enumerate(zip(c, res))]
            b += (4 * u[4] - 2) * g[2].view(-1, 1, 1) * g[1].view(1, -1, 1) * g[0].view(1, 1, -1)
        b += 1e-3 * torch.randn(b.shape, generator=gen, device=DEV)
        b -= b.double().mean().float()
        return {"kind": kind, "solver": F.Poisson(res, 0.005, case["form"]), "b": b, "x": torch.zeros_like(b), "tol": case["tol"]}
    sim = _sim(dict(case, cell=1.2 / case["nx"], spots=5), seed)
    vol = F.Volume(sim, width=case["width"], height=case["height"], vol_scale=case["scale"])
    vol.set_camera((0.75, 0.75, 1.8), (0.0, 0.6, 0.0), 40.0)
    if case["cubic"]:
        vol.set_params({"cubic": 1.0, "flameSharp": case["sharp"]})
    return {"kind": kind, "vol": vol, "frame": 0}


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "step":
        state["sim"].step(state["dt"], 1, stream=_stream())
        return state["out"]
    if kind == "ensemble":
        state["ens"].step(state["dt"], 1, stream=_stream())
        return state["out"]
    if kind == "fit":   # every iteration of a fit starts from the same stored state
        for n, v in state["views"].items():
            v.copy_(state["start"][n])
        adj = state["adj"]
        adj.forward(1 / 120, stream=_stream())
        loss = adj.loss(state["target"])
        adj.backward(stream=_stream())
        grad = adj.grad_spots(state["spots"])   # the fluxes are 32-bit, and so are what the update needs of these
        return {"loss": np.float32(loss), "grad": grad.astype(np.float32), "final": {n: state["views"][n] for n in ("vel", "S", "S2")}}
    if kind == "poisson":
        x = state["x"].zero_()
        state["solver"].solve(state["b"], x, tol=state["tol"], max_iters=40, stream=_stream())
        return x
    state["frame"] += 1
    state["vol"].render(1.0 + state["frame"] / 30.0, state["frame"], stream=_stream())
    return {"image": state["vol"].image(), "lights": state["vol"].lights()}


def _cells(case):
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """A step: vel, S, S2, p in and out (104 bytes a cell) and geometry in (16).  A solve: b in, x out; its
    operations are those of five V(2,2) cycles.  A fit: the stored state, the reverse sweep's reading of what the
    rollout wrote, per step.  A render: S and S2 in, the image out."""
    kind = case["kind"]
    if kind == "step":
        return {"bytes": 120.0 * _cells(case), "flops": (1500.0 + 75.0 * (case["cycles"] if _fixed(case) else 3)) * _cells(case)}
    if kind == "ensemble":
        n = sum(g[0] * g[1] * g[2] for g in _ensemble_grids(case))
        return {"bytes": 120.0 * n, "flops": (1500.0 + 75.0 * case["cycles"]) * n}
    if kind == "fit":
        return {"bytes": 360.0 * case["steps"] * _cells(case), "flops": 6000.0 * case["steps"] * _cells(case)}
    if kind == "poisson":
        return {"bytes": 8.0 * _cells(case), "flops": 375.0 * _cells(case)}
    px = round(case["width"] * case["scale"]) * round(case["height"] * case["scale"])
    return {"bytes": 32.0 * _cells(case) + 16.0 * px, "flops": 100.0 * 150.0 * px}


# ------------------------------------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    if kind == "poisson":
        return _exact_poisson(prepare(case, seed)["b"].double(), 0.005)
    return None   # the fit's gradients and the march through the volume have no short 64-bit form


def _exact_step(case, seed):
    if _cells(case) > 6_000_000:
        return None
    sim = prepare(case, seed)["sim"]
    solve = (case["cycles"], case["tol"], case["omega"])
    return _step64(sim, case["dt"], solve)


def _exact_ensemble(case, seed):
    st = prepare(case, seed)
    return [{n: v for n, v in _step64(s, st["dt"], (case["cycles"], 0.0, 1.0)).items() if n != "p"} for s in st["ens"].members]


def _step64(sim, dt, solve):
    """One simulation step in 64 bits from the simulation's fields, parameter block, noise tables and emitter
    geometry (all taken as inputs)."""
    sim.run_stage("geo", dt, stream=_stream())
    blk = sim.peek_block(dt).astype(np.float64)
    P = dict(zip(F.SIM_FIELDS, blk.tolist()))
    E = blk[64:].tolist()
    get = lambda n: _view(sim, n).double()
    vel, S, S2, geo, p = get("vel")[..., :3], get("S"), get("S2"), get("geo"), get("p")
    hats, tops = _advect(P, vel, S, S2)
    v, phi, S, S2 = _forces(P, E, tops, geo, _view(sim, "noise").double(), _view(sim, "curl").double())
    dx = P["dx"]
    x, y, z = [_shift(v[..., c], c) for c in range(3)]
    below = y[0].clone()
    below[:, 0] = -v[:, 0, :, 1]
    b = ((x[1] - x[0]) + (y[1] - below) + (z[1] - z[0])) / (2 * dx) - phi
    p = _solve(p, b, [(tuple(l["dims"]), l["h"]) for l in sim.levels], sim.coarse_iters, *solve)
    g = []
    for c in range(3):
        lo, hi = _shift(p, c)
        lo, hi = lo.clone(), hi.clone()
        d = 2 - c
        lo.select(d, 0).copy_(p.select(d, 0) * (1 if c == 1 else -1))
        hi.select(d, -1).copy_(-p.select(d, -1))
        g.append((hi - lo) / (2 * dx))
    v = v - torch.stack(g, -1)
    v[geo[..., 2] > 0.5] = 0
    v[:, 0, :, 1].clamp_(min=0)
    length = v.norm(dim=-1, keepdim=True)
    v = torch.where(length > 20, v * 20 / length, v)
    return {"vel": torch.cat([v, torch.zeros_like(length)], -1), "S": S, "S2": S2, "p": p}


def _shift(f, axis):
    """The clamped neighbours of f (z, y, x[, c]) below and above along axis 0 = x, 1 = y, 2 = z."""
    d = 2 - axis
    n = f.shape[d]
    lo = torch.cat([f.narrow(d, 0, 1), f.narrow(d, 0, n - 1)], d)
    hi = torch.cat([f.narrow(d, 1, n - 1), f.narrow(d, n - 1, 1)], d)
    return lo, hi


def _smoothstep(e0, e1, x):
    t = ((x - e0) / (e1 - e0)).clamp(0, 1)
    return t * t * (3 - 2 * t)


def _corner(f, i0, q, dims, repeat=False):
    flat = 0
    for c, n, stride in zip(range(3), dims, (1, dims[0], dims[0] * dims[1])):
        i = i0[c] + ((q >> c) & 1)
        flat = flat + (i % n if repeat else i.clamp(0, n - 1)) * stride
    return f.reshape(-1, f.shape[-1])[flat.reshape(-1)].reshape(flat.shape + f.shape[-1:])


def _sample(f, c, repeat=False):
    """Trilinear sample of f (z, y, x, channels) at cell coordinates c = [x, y, z], clamped or repeating."""
    dims = (f.shape[2], f.shape[1], f.shape[0])
    u = [a - 0.5 for a in c]
    i0 = [a.floor().long() for a in u]
    fr = [a - i for a, i in zip(u, i0)]
    out = 0
    for q in range(8):
        w = 1
        for k in range(3):
            w = w * (fr[k] if (q >> k) & 1 else 1 - fr[k])
        out = out + w[..., None] * _corner(f, i0, q, dims, repeat)
    return out


def _advect(P, vel, S, S2):
    nz, ny, nx, _ = S.shape
    dims, dev = (nx, ny, nz), S.device
    r = [torch.arange(n, device=dev, dtype=torch.float64) + 0.5 for n in dims]
    c = [r[0].view(1, 1, -1).expand(nz, ny, nx), r[1].view(1, -1, 1).expand(nz, ny, nx), r[2].view(-1, 1, 1).expand(nz, ny, nx)]
    k = P["dt"] / P["dx"]
    mid = _sample(vel, [c[i] - 0.5 * k * vel[..., i] for i in range(3)])
    b = [c[i] - k * mid[..., i] for i in range(3)]
    out = torch.maximum(torch.maximum(b[0] - nx, b[1] - ny), b[2] - nz)
    fade = (1 - torch.maximum(-torch.minimum(b[0], b[2]), out)).clamp(0, 1)[..., None]
    ws = _smoothstep(0.03, 0.4, b[1] * P["dx"])
    wind = torch.stack([P["windX"] * ws, 0 * ws, P["windZ"] * ws], -1)
    hats = [wind * (1 - fade) + _sample(vel, b) * fade, _sample(S, b) * fade, _sample(S2, b) * fade]
    fw = [c[i] + k * vel[..., i] for i in range(3)]
    i0 = [(a - 0.5).floor().long() for a in b]
    tops = []
    for f, h in zip((vel, S, S2), hats):
        n = torch.where(fade < 1, h, h + 0.5 * (f - _sample(h, fw)))
        lo, hi = h, h
        for q in range(8):
            t = _corner(f, i0, q, dims)
            lo, hi = torch.minimum(lo, t), torch.maximum(hi, t)
        n = torch.minimum(torch.maximum(n, lo), hi)
        tops.append(n if f is vel else n.clamp(min=0))
    return hats, tops


def _curl(v):
    x, y, z = _shift(v, 0), _shift(v, 1), _shift(v, 2)
    d = [hi - lo for lo, hi in (x, y, z)]
    return 0.5 * torch.stack([d[1][..., 2] - d[2][..., 1], d[2][..., 0] - d[0][..., 2], d[0][..., 1] - d[1][..., 0]], -1)


def _forces(P, E, tops, geo, noise, curl):
    """Sources, combustion, soot, cooling, buoyancy, confinement, curl noise, wind and sponge.  E: soot age gate
    (0, 1), bed gain, spot count and reference flux (3, 4), spots from 16 on, eight numbers each."""
    v, S, S2 = tops
    nz, ny, nx, _ = S.shape
    dt, dx, I = P["dt"], P["dx"], P["intensity"]
    idx = [torch.arange(n, device=v.device, dtype=torch.float64) + 0.5 for n in (nx, ny, nz)]
    full = lambda a: a.expand(nz, ny, nx)
    px, py, pz = full(P["ox"] + dx * idx[0].view(1, 1, -1)), full(P["oy"] + dx * idx[1].view(1, -1, 1)), full(P["oz"] + dx * idx[2].view(-1, 1, 1))
    lookup = lambda tab, q: _sample(tab, [a * tab.shape[0] for a in q], repeat=True)
    band, bedg, solid = geo[..., 0], geo[..., 1], geo[..., 2]
    T, fuel, soot, heat = S.unbind(-1)
    prod, age, smoke, co = S2.unbind(-1)
    on = band > 0.001
    ka, kn = P["anchorFreq"], P["srcFreq"] * 0.06
    anchor = _smoothstep(-0.05, 0.25, 2 * lookup(noise, [px * ka + P["seed"] * 0.37, py * ka, pz * ka + 0.11])[..., 2] - 1) * on
    th = P["srcThresh"]
    pulse = _smoothstep(th - 0.25, th + 0.25, 2 * lookup(noise, [px * kn + P["seed"] * 0.131, py * kn, pz * kn + P["time"] * P["srcSpeed"]])[..., 0] - 1)
    src = (band * P["logSrc"] * (P["srcFloor"] + P["anchorGain"] * anchor) * (0.55 * (1 - pulse) + pulse) * 1.2).clamp(0, 1) * I * (1 - solid) * on
    acc = torch.zeros_like(T)
    for q in range(int(E[3])):
        sx, sy, sz, sg, fl = E[16 + 8 * q:21 + 8 * q]
        d2 = (px - sx) ** 2 + (py - sy) ** 2 + (pz - sz) ** 2
        acc += (fl / E[4]) * torch.exp(-d2 / (2 * sg * sg)) * (d2 < 16 * sg * sg)
    src = torch.maximum(src, acc.clamp(0, 1) * I)
    srcW = src.clamp(max=1)
    bed = bedg * min(max(I * 1.4, 0.3), 1.0)
    qb = [px * 2.4 + 0.17, py * 2.4 - P["time"] * 0.12, pz * 2.4 + P["time"] * 0.05]
    bed = torch.where(bed > 0.001, bed * _smoothstep(0, 0.3, 2 * lookup(noise, qb)[..., 1] - 1), bed)
    fuel = torch.maximum(torch.maximum(fuel, src * P["fuelSrc"]), bed * P["bedFuel"])
    T = torch.maximum(torch.maximum(T, src * P["srcTemp"]), bedg * P["bedTemp"])
    srcAll = torch.maximum(srcW, bed)
    t1 = bed * (1 - srcW)
    co = (co * (1 - t1) + t1) * (1 - srcW)
    age = age * (1 - srcAll)
    prod = torch.maximum(torch.maximum(prod, (1 - fuel) * srcW), (1 - fuel) * bed * 0.6)
    wsrc = 1 - (1 - 0.5 * (srcW + 0.4 * bed).clamp(0, 1)) ** (dt * 90)
    vx, vy, vz = v.unbind(-1)
    vy = vy * (1 - wsrc) + vy.clamp(min=P["srcVel"]) * wsrc
    smoke = smoke + band * (1 - anchor) * P["smolder"] * dt * I
    ageF = age / (fuel + prod).clamp(min=1e-4)
    T0 = 293 + 1000 * T
    o = (1 - fuel - prod).clamp(0, 1)
    ign = _smoothstep(P["ignT"] - 50, P["ignT"] + 50, T0)
    b = torch.minimum(fuel, o / P["rs"]) * (1 - torch.exp(-P["kMix"] * ign * dt))
    fuel = fuel - b
    prod = (prod + (1 + P["rs"]) * b).clamp(max=1)
    dT = torch.minimum(P["heatOut"] * b, (2100 - T0).clamp(min=0))
    T = T0 + dT
    q = dT / dt
    phi = torch.where(solid > 0.5, torch.zeros_like(q), (P["expansion"] * q / T).clamp(max=60))
    ageF = (ageF + dt).clamp(max=4)
    soot = soot + P["sootForm"] * b * _smoothstep(E[0], E[1], ageF) * _smoothstep(1000, 1400, T) * (1 - co)
    ox = P["sootOx"] * dt
    soot = soot * torch.exp(-ox * (0.25 + o) * _smoothstep(1100, 1400, T))
    soot = soot * torch.exp(-ox * 0.5 * o * _smoothstep(850, 1100, T) * (1 - _smoothstep(1100, 1300, T))) * math.exp(-P["sootDissip"] * dt)
    tk = T * 0.001
    T = T - (P["radCool"] * 970 * soot * tk * tk * (tk ** 4 - 0.00737)).clamp(max=6000) * dt
    T = 293 + (T - 293).clamp(min=0) * torch.exp(-P["coolRate"] * (1 - _smoothstep(500, 5000, q)) * dt)
    theta, heat = (T - 293) * 0.001, q * 1e-4
    fuel, prod, smoke = fuel * math.exp(-P["fuelDissip"] * dt), prod * math.exp(-P["vitDecay"] * dt), smoke * math.exp(-P["smokeDissip"] * dt)
    age = ageF * (fuel + prod).clamp(0, 1)
    v = torch.stack([vx, vy + P["buoyancy"] * theta * dt, vz], -1)
    w = _curl(tops[0])
    wl = w.norm(dim=-1)
    g = torch.stack([hi - lo for lo, hi in (_shift(wl, 0), _shift(wl, 1), _shift(wl, 2))], -1)
    gl = g.norm(dim=-1, keepdim=True)
    gate = _smoothstep(450, 900, T) * (1 - srcAll) * _smoothstep(0.02, 0.08, py)
    n = torch.where(gl > 1e-6, g / gl.clamp(min=1e-30), torch.zeros_like(g))
    v = v + torch.cross(n, w, dim=-1) * (P["vortEps"] * gate * dt)[..., None]
    tgate = torch.maximum(_smoothstep(500, 1100, T), _smoothstep(0, 3, heat)) * (1 - srcAll) * (0.6 + 1.2 * _smoothstep(0.2, 0.75, py))
    tf, time = P["turbFreq"], P["time"]
    cn = lookup(curl, [px * tf, (py - time * P["turbRise"]) * tf, pz * tf + time * P["turbEvolve"]])[..., :3]
    v = v + cn * (P["turbAmp"] / 12 * tgate * dt * 10)[..., None]
    windK = _smoothstep(0.05, 0.5, py) * (1 + P["gust"])
    wsy = _smoothstep(0.03, 0.4, py)
    side = torch.minimum(torch.minimum(idx[0], nx - idx[0]).view(1, 1, -1), torch.minimum(idx[2], nz - idx[2]).view(-1, 1, 1)).expand(nz, ny, nx)
    ks = 1 - (1 - 0.15 * ((1 - _smoothstep(0, 5, side)) * P["sponge"]).clamp(0, 1)) ** (dt * 90)
    parts = []
    for i, wind in enumerate((P["windX"], None, P["windZ"])):
        a = v[..., i]
        if wind is not None:
            a = a + (wind * windK - a) * dt * 0.35 * windK
        a = a * math.exp(-P["velDissip"] * dt) * (solid <= 0.5)
        parts.append(a if wind is None else a * (1 - ks) + wind * wsy * ks)
    v = torch.stack(parts, -1)
    fuel, age = fuel * (solid <= 0.5), age * (solid <= 0.5)
    kt = ((1 - 0.1 * _smoothstep(ny - 10.0, float(ny), idx[1])) ** (dt * 90)).view(1, -1, 1)
    length = v.norm(dim=-1, keepdim=True)
    v = torch.where(length > 15, v * 15 / length, v)
    return v, phi, torch.stack([theta, fuel, soot * kt, heat], -1), torch.stack([prod, age, smoke * kt, co], -1)


# The multigrid solve: red-black sweeps, residual restriction over 8 children, trilinear prolongation.  Open
# sides and top (ghost -p), solid floor (ghost p): both fold into the diagonal.
def _inside_sum(p):
    s = torch.zeros_like(p)
    for d in range(3):
        n = p.shape[d]
        s.narrow(d, 1, n - 1).add_(p.narrow(d, 0, n - 1))
        s.narrow(d, 0, n - 1).add_(p.narrow(d, 1, n - 1))
    return s


def _diag(p):
    d = torch.full_like(p, 6.0)
    for axis in range(3):
        d.select(axis, 0).add_(-1.0 if axis == 1 else 1.0)
        d.select(axis, -1).add_(1.0)
    return d


def _sweeps(p, b, h, n, omega):
    diag = _diag(p)
    parity = sum(torch.arange(p.shape[d], device=p.device).view([-1 if e == d else 1 for e in range(3)]) for d in range(3)) % 2
    for k in range(2 * n):
        gs = (_inside_sum(p) - h * h * b) / diag
        p = torch.where(parity == k % 2, p + omega * (gs - p), p)
    return p


def _residual(p, b, h):
    return b - (_inside_sum(p) - _diag(p) * p) / (h * h)


def _prolong(c):
    """Twice as many cells along every axis; ghosts: -c beyond the sides and the top, c below the floor."""
    for d in range(3):
        n = c.shape[d]
        first, last = c.narrow(d, 0, 1), c.narrow(d, n - 1, 1)
        e = torch.cat([first if d == 1 else -first, c, -last], d)
        lo = 0.25 * e.narrow(d, 0, n) + 0.75 * c
        hi = 0.75 * c + 0.25 * e.narrow(d, 2, n)
        c = torch.stack([lo, hi], d + 1).flatten(d, d + 1)
    return c


def _cycle(p, b, levels, coarse, omega, l=0):
    (nx, ny, nz), h = levels[l]
    if l == len(levels) - 1:
        return _sweeps(p, b, h, coarse, omega)
    p = _sweeps(p, b, h, 2, omega)
    r = _residual(p, b, h).reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).mean(dim=(1, 3, 5))
    p = p + _prolong(_cycle(torch.zeros_like(r), r, levels, coarse, omega, l + 1))
    return _sweeps(p, b, h, 2, omega)


def _solve(p, b, levels, coarse, cycles, tol, omega):
    for _ in range(cycles):
        p = _cycle(p, b, levels, coarse, omega)
        if tol and _residual(p, b, levels[0][1]).norm() <= tol * b.norm():
            break
    return p


def _exact_poisson(b, h):
    """The solution itself: the operator is a sum over the axes, so it is diagonal in the axes' eigenvectors."""
    lam = 0
    vecs = []
    for d in range(3):
        n = b.shape[d]
        a = torch.diag(torch.full((n - 1,), 1.0, dtype=torch.float64), 1)
        a = a + a.T - 2 * torch.eye(n, dtype=torch.float64)
        a[0, 0] += 1.0 if d == 1 else -1.0
        a[-1, -1] -= 1.0
        w, u = torch.linalg.eigh(a)
        lam = lam + w.to(b.device).view([-1 if e == d else 1 for e in range(3)])
        vecs.append(u.to(b.device))
    x = b * (h * h)
    for d in range(3):
        x = torch.tensordot(x, vecs[d], dims=([0], [0]))   # the transformed axis moves to the back
    x = x / lam
    for d in range(3):
        x = torch.tensordot(x, vecs[d], dims=([0], [1]))
    return x
