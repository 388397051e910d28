"""The work that users have this package do, as measurable cases: single timesteps, whole runs, batches of uneven
problems and gradient evaluations, each through the public Python API.

A case is a dict of plain values.  Its kind:

``step``      one ``run_adi_steps`` call, on a numpy array (as the reference's time loops make it) or a CUDA tensor
``run``       ``run``: nsteps on the device in one call, recording nothing, a layer or the surface estimate
``batch``     ``Batch.run`` of uneven instances and ``get_temperature``, FP64 or FP32
``adjoint``   loss and gradients with respect to k, rho*c, q and T0 of one instance (``surface_misfit``) or of a
              batch (``batch_surface_misfit``), with or without face classes and fixed voxels

Problems come from ``heatsim2_gb300.workloads``: steel slabs (1 mm cells, one thin-layer flaw), composite panels
over aluminium (0.5 mm cells, insulating delaminations, an ambient layer), uneven batches of both, lognormal and
two-phase conductivities.  A forward problem starts from a field some steps after a flash: 293 K, a decaying
profile in depth with smooth lateral variation, and the ambient layer at 293 K.
"""
import math

import numpy as np
import torch

import heatsim2_gb300 as hs
from heatsim2_gb300 import workloads as W
from heatsim2_gb300.adjoint import batch_surface_misfit, surface_misfit
from heatsim2_gb300.batch import Batch


def listed():
    return [
        # the reference demos' own time loop: one step of the small steel slab, numpy in, numpy out
        {"name": "step_slab_host", "kind": "step", "problem": "steel", "nz": 20, "ny": 40, "nx": 40, "host": True},
        # the same loop with the field kept on the device, on a mid-size panel with odd rows
        {"name": "step_panel_device", "kind": "step", "problem": "composite", "nz": 33, "ny": 150, "nx": 171,
         "host": False},
        # a numpy time loop on a large panel: the copies of T to and from the device count
        {"name": "step_panel_host", "kind": "step", "problem": "composite", "nz": 49, "ny": 220, "nx": 200,
         "host": True},
        # the standard small job: 200 steps of the steel slab with the surface temperature recorded each step
        {"name": "run_slab", "kind": "run", "problem": "steel", "nz": 20, "ny": 40, "nx": 40, "nsteps": 200,
         "record": "surface"},
        # a specimen of ordinary size, odd in every direction, one layer recorded
        {"name": "run_panel_odd", "kind": "run", "problem": "composite", "nz": 37, "ny": 187, "nx": 211, "nsteps": 60,
         "record": "layer"},
        # a curved steel part (curvature mode, one factorisation per row)
        {"name": "run_curved", "kind": "run", "problem": "curved", "nz": 24, "ny": 96, "nx": 128, "nsteps": 80,
         "record": "surface"},
        # the large panel, 64x512x512 computed voxels and the ambient layer
        {"name": "run_panel_large", "kind": "run", "problem": "composite", "nz": 65, "ny": 512, "nx": 512,
         "nsteps": 20, "record": "none"},
        # parameter studies: uneven slabs and panels advanced together, in double and in float
        {"name": "batch_fp64", "kind": "batch", "n": 12, "sizes": 2, "nsteps": 200, "precision": 64},
        {"name": "batch_fp32", "kind": "batch", "n": 12, "sizes": 2, "nsteps": 200, "precision": 32},
        # inverse problems: gradients of the surface misfit; a small part with a flaw and a fixed layer, the
        # single steel block, a batch of uneven two-phase specimens
        {"name": "adjoint_flaw_small", "kind": "adjoint", "n": 1, "nz": 12, "ny": 40, "nx": 44, "nsteps": 40,
         "ckpt": 10, "faces": True},
        {"name": "adjoint_steel", "kind": "adjoint", "n": 1, "nz": 32, "ny": 128, "nx": 128, "nsteps": 100,
         "ckpt": 20, "faces": False},
        {"name": "adjoint_batch", "kind": "adjoint", "n": 6, "sizes": 4, "nsteps": 40, "ckpt": 10, "faces": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "run", "run", "run", "batch", "batch", "adjoint", "adjoint", "adjoint"])
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(5, 12), "sizes": rng.randint(0, 999), "nsteps": rng.randint(80, 160),
                "precision": rng.choice([64, 32])}
    if kind == "adjoint" and rng.random() < 0.34:
        return {"kind": "adjoint", "n": rng.randint(2, 6), "sizes": rng.randint(0, 999), "nsteps": rng.randint(16, 40),
                "ckpt": rng.randint(5, 20), "faces": False}
    ny, nx = _log_int(rng, 32, 512), _log_int(rng, 32, 512)
    nz = _log_int(rng, 12, 64)
    if kind == "adjoint":
        ny, nx, nz = min(ny, 200), min(nx, 200), min(nz, 40)
        return {"kind": "adjoint", "n": 1, "nz": nz, "ny": ny, "nx": nx, "nsteps": rng.randint(30, 90),
                "ckpt": rng.randint(8, 30), "faces": rng.random() < 0.4}
    problem = rng.choice(["steel", "composite", "composite"])
    if kind == "step":
        return {"kind": "step", "problem": problem, "nz": nz, "ny": ny, "nx": nx, "host": rng.random() < 0.5}
    if rng.random() < 0.2 and nz * ny * nx < 1 << 20:
        problem = "curved"
    steps = max(15, min(200, int(3e8 / (nz * ny * nx))))
    return {"kind": "run", "problem": problem, "nz": nz, "ny": ny, "nx": nx, "nsteps": steps,
            "record": rng.choice(["none", "layer", "surface"])}


# ---- inputs ----------------------------------------------------------------------------------------------
def _spec(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    if case["problem"] == "composite":
        return W.composite_panel(seed=seed, nz=nz - 1, ny=ny, nx=nx, top_layers=max(1, (nz - 1) // 4),
                                 width_range=(max(3, min(ny, nx) // 16), max(4, min(ny, nx) // 6)),
                                 depth_range=(2, max(3, (nz - 1) * 5 // 8)))
    spec = W.steel_slab(seed=seed, nz=nz, ny=ny, nx=nx, flaw=max(4, min(ny, nx) // 5), depth_range=(3, 3 * nz // 4))
    if case["problem"] == "curved":
        spec = W.curved(spec, ky=2.0 + 0.1 * (seed % 7), kx=1.0)
    return spec


def _field(shape, rng, ambient):
    """293 K plus the remains of a flash: a few kelvin at the top, decaying in depth, smooth across the surface."""
    nz, ny, nx = shape
    y = np.linspace(0.0, 1.0, ny)[:, None]
    x = np.linspace(0.0, 1.0, nx)[None, :]
    lat = np.ones((ny, nx))
    for _ in range(4):
        fy, fx, ph, a = rng.uniform(0.5, 6.0), rng.uniform(0.5, 6.0), rng.uniform(0, 6.28), rng.uniform(0.02, 0.12)
        lat = lat + a * np.sin(2 * np.pi * (fy * y + fx * x) + ph)
    depth = np.exp(-np.arange(nz) / (0.15 * nz + 1.0)) * rng.uniform(2.0, 6.0)
    T = 293.0 + depth[:, None, None] * lat[None]
    if ambient:
        T[0] = 293.0
    return T


def _sizes(case, nz_range, nxy_range):
    """The batch's grid shapes: uneven, fixed by the case (the seed of the inputs draws what is in them)."""
    rng = np.random.default_rng(case["sizes"])
    return [tuple(int(rng.integers(lo, hi + 1)) for lo, hi in (nz_range, nxy_range, nxy_range))
            for _ in range(case["n"])]


def _batch_specs(case, seed):
    """Slabs and panels in turn, a flaw 4..32 voxels wide at a depth of 2..nz/2, 10 ms steps."""
    rng = np.random.default_rng(seed)
    specs = []
    for i, (nz, ny, nx) in enumerate(_sizes(case, (16, 64), (64, 256))):
        w, sub, depth = int(rng.integers(4, 33)), int(rng.integers(0, 2 ** 31)), (2, max(2, nz // 2))
        if i % 2 == 0:
            specs.append(W.steel_slab(seed=sub, nz=nz, ny=ny, nx=nx, flaw=w, depth_range=depth))
        else:
            specs.append(W.composite_panel(seed=sub, nz=nz, ny=ny, nx=nx, dt=0.01, n_delams=1, width_range=(w, w),
                                           depth_range=depth, power=1e9))
    return specs


def _adjoint_problems(case, seed):
    if "nz" in case:
        p = W.adjoint_steel(seed=seed, nz=case["nz"], ny=case["ny"], nx=case["nx"], nsteps=case["nsteps"],
                            ckpt=case["ckpt"])
        if case["faces"]:
            nz, ny, nx = p["shape"]
            s = W.steel_slab(seed=seed, nz=nz, ny=ny, nx=nx, flaw=max(3, min(ny, nx) // 4), depth_range=(2, nz // 2))
            p["spec"] = s
            fixed = np.zeros(p["shape"], dtype=bool)
            fixed[-1] = True
            p["fixed"] = fixed
        return [p]
    rng = np.random.default_rng(seed)
    out = []
    schedule = np.zeros(case["nsteps"])
    schedule[0] = 1.0
    for shape in _sizes(case, (24, 48), (96, 192)):
        C, q = 1550.0 * 1100.0, np.zeros(shape)
        q[0] = 2e9
        out.append({"shape": shape, "spacing": (0.5e-3,) * 3, "dt": 0.005, "k": W.two_phase_k(rng, shape),
                    "C": np.full(shape, C), "q": q, "T0": np.full(shape, W.T_AMBIENT), "schedule": schedule,
                    "obs": W.flash_observations(rng, shape, case["nsteps"], 0.005, 0.5e-3, 5.0, C, 2e9)})
    return out


def _faces(p):
    if "spec" not in p:
        return None
    a = p["spec"]["arrays"]
    return (W.boundaries_tuple(hs, p["spec"]), a["boundary_z"], a["boundary_y"], a["boundary_x"])


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1000)
    if kind in ("step", "run"):
        spec = _spec(case, seed)
        P, S = hs.setup(*W.setup_args(hs, spec), **W.setup_kwargs(spec))
        T = _field((case["nz"], case["ny"], case["nx"]), rng, case["problem"] == "composite")
        host = case.get("host", False)
        return {"case": case, "spec": spec, "P": P, "S": S, "vol": W.volumetric_tuple(hs, spec),
                "T": T if host else torch.from_numpy(T).cuda(), "times": W.step_times(spec, case.get("nsteps", 1))}
    if kind == "batch":
        specs = _batch_specs(case, seed)
        b = Batch([W.setup_args(hs, s) for s in specs], precision=case["precision"])
        b.set_temperature([_field(b.shapes[i], rng, s["name"] == "composite_panel") for i, s in enumerate(specs)])
        b.set_sources(W.step_times(specs[0], 1), specs[0]["dt"])      # the flash fires in the first step
        return {"case": case, "batch": b}
    ps = _adjoint_problems(case, seed)
    dev = [{n: torch.from_numpy(p[n]).cuda() for n in ("k", "C", "q", "T0", "obs")} for p in ps]
    for d in dev:
        for n in ("k", "C", "q", "T0"):
            d[n].requires_grad_()
    return {"case": case, "ps": ps, "dev": dev, "faces": [_faces(p) for p in ps]}


# ---- one pass --------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        # a step of the time loop after the flash has ended (no source is active)
        spec = state["spec"]
        return hs.run_adi_steps(state["P"], state["S"], 5 * spec["dt"], spec["dt"], state["T"],
                                spec["arrays"]["volumetric"], state["vol"])
    if kind == "run":
        spec = state["spec"]
        kw = {"none": {}, "layer": {"record_layer": 1}, "surface": {"record_surface": True}}[case["record"]]
        return hs.run(state["P"], state["T"], state["times"], spec["dt"], spec["arrays"]["volumetric"], state["vol"],
                      **kw)
    if kind == "batch":
        state["batch"].run(case["nsteps"])
        return state["batch"].get_temperature()
    dev, ps = state["dev"], state["ps"]
    leaves = [d[n] for d in dev for n in ("k", "C", "q", "T0")]
    if len(dev) == 1:
        d, p = dev[0], ps[0]
        loss = surface_misfit(d["k"], d["C"], d["q"], d["T0"], d["obs"], p["schedule"], p["spacing"], p["dt"],
                              case["ckpt"], state["faces"][0], p.get("fixed"))
        return [loss.detach()] + list(torch.autograd.grad(loss, leaves))
    loss = batch_surface_misfit([d["k"] for d in dev], [d["C"] for d in dev], [d["q"] for d in dev],
                                [d["T0"] for d in dev], [d["obs"] for d in dev], ps[0]["schedule"],
                                [p["spacing"] for p in ps], ps[0]["dt"], case["ckpt"])
    return [loss.detach()] + list(torch.autograd.grad(loss.sum(), leaves))


# ---- what a pass cannot do without -----------------------------------------------------------------------
# Forward: per voxel and step T is read and written and 14 fused multiply-adds are done (a seven-point stencil, two
# recurrences per line solve, the update); the class maps (material, source and three boundary arrays, a byte each)
# are read once per pass.  Gradients: per voxel and step the forward pass keeps T, the reverse pass reads it and
# updates the adjoint state and the accumulated gradients; 79 multiply-adds with the recompute.
def work(case):
    kind = case["kind"]
    if kind in ("step", "run"):
        n, steps = case["nz"] * case["ny"] * case["nx"], case.get("nsteps", 1)
        rec = 0 if case.get("record", "none") == "none" else 8 * steps * case["ny"] * case["nx"]
        return {"bytes": 16 * n + 5 * n + rec, "flops": 28 * n * steps}
    if kind == "batch":
        n = sum(a * b * c for a, b, c in _sizes(case, (16, 64), (64, 256)))
        e = case["precision"] // 8
        return {"bytes": (2 * e + 5 + 8) * n, "flops": 28 * n * case["nsteps"]}
    shapes = [(case["nz"], case["ny"], case["nx"])] if "nz" in case else _sizes(case, (24, 48), (96, 192))
    n, top = sum(a * b * c for a, b, c in shapes), sum(b * c for _, b, c in shapes)
    return {"bytes": 8 * 8 * n + 8 * top * case["nsteps"], "flops": 158 * n * case["nsteps"]}


# ---- the same results in plain torch, 64 bits ------------------------------------------------------------
def _shift(a, s, dim, fill=0.0):
    """a moved by s along dim (value at index i comes from i - s), fill where there is none."""
    n = a.shape[dim]
    if abs(s) >= n:
        return torch.full_like(a, fill)
    pad = torch.full_like(a.narrow(dim, 0, abs(s)), fill)
    return torch.cat([pad, a.narrow(dim, 0, n - s)] if s > 0 else [a.narrow(dim, -s, n + s), pad], dim)


class _Lines(object):
    """Tridiagonal solves along dim by parallel cyclic reduction, the reduction coefficients formed once."""

    def __init__(self, lo, d, hi, dim):
        self.dim, self.levels = dim, []
        s = 1
        while s < d.shape[dim]:
            k1 = lo / _shift(d, s, dim, 1.0)
            k2 = hi / _shift(d, -s, dim, 1.0)
            self.levels.append((s, k1, k2))
            d = d - k1 * _shift(hi, s, dim) - k2 * _shift(lo, -s, dim)
            lo, hi = -k1 * _shift(lo, s, dim), -k2 * _shift(hi, -s, dim)
            s *= 2
        self.d = d

    def solve(self, f):
        for s, k1, k2 in self.levels:
            f = f - k1 * _shift(f, s, self.dim) - k2 * _shift(f, -s, self.dim)
        return f / self.d


class _Model(object):
    """The Douglas step (M - La/2) per axis from per-row face conductances glo, ghi (zero rows where fixed)."""

    def __init__(self, glo, ghi, M, comp):
        self.glo = [g * comp for g in glo]
        self.ghi = [g * comp for g in ghi]
        self.M, self.comp = torch.where(comp > 0, M, torch.ones_like(M)), comp
        self.lines = [_Lines(-l / 2, self.M + (l + h) / 2, -h / 2, a) for a, (l, h) in enumerate(zip(self.glo, self.ghi))]

    def step(self, T, q=None):
        r = torch.zeros_like(T)
        for a in range(3):
            r = r + self.glo[a] * (_shift(T, 1, a) - T) + self.ghi[a] * (_shift(T, -1, a) - T)
        if q is not None:
            r = r + q * self.comp
        for a in (2, 1, 0):
            r = self.lines[a].solve(r if a == 2 else self.M * r)
        return T + r


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _class_model(spec, device):
    """_Model of a class problem: every built-in boundary class is const * (T_hi - T_lo) with const = mean k / d
    (conducting, with the axis's own tensor entry) or h; flat cells, or the cells of a curved surface."""
    a, g = spec["arrays"], spec["grid"]
    d = (g["dz"], g["dy"], g["dx"])
    mat = torch.from_numpy(a["material"]).long().to(device)
    kt = np.zeros((len(spec["materials"]), 3))
    cap = np.ones(len(spec["materials"]))
    for m, e in enumerate(spec["materials"]):
        if e[0] == "compute":
            kt[m] = [e[1][i][i] for i in range(3)] if isinstance(e[1], list) else [e[1]] * 3
            cap[m] = e[2] * e[3] / spec["dt"]
    comp_m = torch.tensor([float(e[0] == "compute") for e in spec["materials"]], dtype=torch.float64, device=device)
    comp = comp_m[mat]
    shape = mat.shape
    k = torch.arange(shape[0], dtype=torch.float64, device=device)[:, None, None]
    zero = torch.zeros(shape[1:], dtype=torch.float64, device=device)
    curv = [torch.from_numpy(np.asarray(a[n])).to(device) if n in a else zero for n in ("curv_y", "curv_x")]
    top = [(1 + k * c[None] * d[0]) * e for c, e in zip(curv, d[1:])]
    bot = [(1 + (k + 1) * c[None] * d[0]) * e for c, e in zip(curv, d[1:])]
    dy, dx = [(t + b) / 2 for t, b in zip(top, bot)]
    vol = (dx * dy * d[0]).abs()
    edge = (torch.full_like(dy, d[0]), dy, dx)
    area = (((top[0] * top[1]), (bot[0] * bot[1])), (dx * d[0],) * 2, (dy * d[0],) * 2)
    glo, ghi = [], []
    for ax, key in enumerate(("boundary_z", "boundary_y", "boundary_x")):
        ka = torch.from_numpy(kt[:, ax].copy()).to(device)[mat]
        cls = torch.from_numpy(a[key]).long().to(device)
        for side, out in ((0, glo), (1, ghi)):
            s = 1 if side == 0 else -1
            has = _shift(comp, s, ax) > 0
            kn = torch.where(has, _shift(ka, s, ax), ka)        # a fixed neighbour lends the cell's own k
            c = cls.narrow(ax, side, shape[ax])
            F = torch.zeros(shape, dtype=torch.float64, device=device)
            for b, e in enumerate(spec["boundaries"]):
                if e[0] in ("conducting", "conducting_anisotropic"):
                    F = torch.where(c == b, (ka + kn) / 2 / edge[ax], F)
                elif e[0] == "thininsulatinglayer":
                    F = torch.where(c == b, torch.full_like(F, float(e[1])), F)
            out.append(area[ax][side] * F / vol)
    M = torch.from_numpy(cap).to(device)[mat]
    q = None
    for c, e in enumerate(spec["volumetric"]):
        if e[0] == "stepped":
            q = (torch.from_numpy(a["volumetric"]).to(device) == c).double() * float(e[3])
    return _Model(glo, ghi, M, comp), q


def _advance(spec, T, t, device, record=None):
    model, q = _class_model(spec, device)
    src = [e for e in spec["volumetric"] if e[0] == "stepped"][0]
    dz2 = spec["grid"]["dz"] ** 2
    hist = []
    for tn in t:
        T = model.step(T, q if src[1] <= tn <= src[2] else None)
        if record == "layer":
            hist.append(T[1])
        elif record == "surface":
            a = (T[1] - T[0]) / (2 * dz2)
            hist.append(((T[0] - (T[1] - T[0]) / 2) + (T[0] - 0.25 * a * dz2)) / 2)
    return T, hist


def _misfit(p, leaf, device):
    """The misfit of one instance by autograd through the plain model."""
    k, C, q, T, obs = (leaf[n] for n in ("k", "C", "q", "T0", "obs"))
    fixed = torch.zeros(p["shape"], dtype=torch.bool) if "fixed" not in p else torch.from_numpy(p["fixed"])
    comp = (~fixed).double().to(device)
    glo, ghi = [], []
    for ax, key in enumerate(("boundary_z", "boundary_y", "boundary_x")):
        n, d = p["shape"][ax], p["spacing"][ax]
        for side, out in ((0, glo), (1, ghi)):
            s = 1 if side == 0 else -1
            inside = _shift(torch.ones_like(comp), s, ax)
            has = _shift(comp, s, ax) > 0
            G = (k + torch.where(has, _shift(k, s, ax), k)) / 2 / (d * d)
            if "spec" in p:
                c = torch.from_numpy(p["spec"]["arrays"][key]).to(device).narrow(ax, side, n)
                for b, e in enumerate(p["spec"]["boundaries"]):
                    if e[0] == "insulating":
                        G = torch.where(c == b, torch.zeros_like(G), G)
                    elif e[0] == "thininsulatinglayer":
                        G = torch.where(c == b, torch.full_like(G, e[1] / d), G)
            out.append(G * inside)
    model = _Model(glo, ghi, C / p["dt"], comp)
    J = 0.0
    for n, s in enumerate(p["schedule"]):
        T = model.step(T, s * q)
        J = J + ((T[0] - obs[n]) ** 2).sum()
    return J


def exact(case, seed):
    device = _device()
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1000)
    if kind in ("step", "run"):
        spec = _spec(case, seed)
        T = torch.from_numpy(_field((case["nz"], case["ny"], case["nx"]), rng, case["problem"] == "composite")).to(device)
        t = W.step_times(spec, case.get("nsteps", 1)) if kind == "run" else [5 * spec["dt"]]
        T, hist = _advance(spec, T, t, device, case.get("record"))
        if kind == "step":
            return T.cpu().numpy() if case["host"] else T
        return T if case["record"] == "none" else (T, torch.stack(hist))
    if kind == "batch":
        specs = _batch_specs(case, seed)
        fields = [_field(s["arrays"]["material"].shape, rng, s["name"] == "composite_panel") for s in specs]
        return [_advance(s, torch.from_numpy(T).to(device), W.step_times(s, case["nsteps"]), device)[0].cpu().numpy()
                for s, T in zip(specs, fields)]
    losses, grads = [], []
    for p in _adjoint_problems(case, seed):
        leaf = {n: torch.from_numpy(p[n]).to(device) for n in ("k", "C", "q", "T0", "obs")}
        at = [leaf[n].requires_grad_() for n in ("k", "C", "q", "T0")]
        J = _misfit(p, leaf, device)
        grads += list(torch.autograd.grad(J, at))
        losses.append(J.detach())
    return [losses[0] if case["n"] == 1 else torch.stack(losses)] + grads
