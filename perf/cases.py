"""The work that users of nhwave_gb300 have it do, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (a scenario set up on the GPU and pinned host buffers for its output),
``run`` makes one pass through the public entry points.  Sizes are those of the
five configurations of ``nhwave_gb300/scenarios.py`` and ragged ones between
them.

The FP64 form is the parity form, so its cases solve the pressure to the
tolerance that the parity tests use (1e-12), and its fields come back as FP64.
The FP32+IR form is the production form, with the configurations' tolerance
1e-8; it keeps U, V, W in single precision and a program writes its output in
single precision, so its fields come back as FP32.
"""
import math
import random

import numpy as np
import torch

from nhwave_gb300 import fields as F
from nhwave_gb300 import lib, scenarios
from nhwave_gb300.params import default_params

FP64, FP32 = 0, 1
G = float(np.float32(9.81))
STATE = ("ETA", "U", "V", "W", "P")
FLUXES = ("EX", "FX", "GX", "HX", "EY", "FY", "GY", "HY", "FZ", "GZ", "HZ")


def listed():
    return [
        # a host model's own arrays on the GPU, one time step asked of them: the smallest call there is
        {"name": "dt_device_arrays", "kind": "dt", "M": 256, "N": 8, "K": 10},
        # partial integration: a driver takes the fluxes alone and keeps the rest of its step
        {"name": "fluxes_ragged_fp32", "kind": "fluxes", "M": 333, "N": 61, "K": 13, "precision": FP32},
        # the solitary wave in a channel, the smallest whole run (launches and latency)
        {"name": "channel_fp64", "kind": "run", "scene": "channel", "M": 256, "N": 8, "K": 10, "precision": FP64,
         "steps": 4},
        {"name": "channel_fp32", "kind": "run", "scene": "channel", "M": 256, "N": 8, "K": 10, "precision": FP32,
         "steps": 8},
        # the monochromatic wave over a submerged bar, the headline run, in both forms
        {"name": "bar_fp32", "kind": "run", "scene": "bar", "M": 1024, "N": 64, "K": 20, "precision": FP32, "steps": 4},
        {"name": "bar_fp64", "kind": "run", "scene": "bar", "M": 1024, "N": 64, "K": 20, "precision": FP64, "steps": 1},
        # the landslide over a wet/dry beach
        {"name": "beach_fp32", "kind": "run", "scene": "beach", "M": 512, "N": 512, "K": 10, "precision": FP32,
         "steps": 2},
        # the same, odd sizes, called routine by routine as the Fortran driver calls the drop-in
        {"name": "beach_routines_ragged_fp64", "kind": "routines", "scene": "beach", "M": 263, "N": 187, "K": 9,
         "precision": FP64, "steps": 1},
        # one large basin with an uneven bed: the largest run
        {"name": "basin_large_fp32", "kind": "run", "scene": "basin", "M": 768, "N": 768, "K": 20, "precision": FP32,
         "steps": 1},
        # an ensemble of uneven basins advanced together
        {"name": "ensemble_fp32", "kind": "ensemble", "members": 12, "sizes": 7, "side_lo": 64, "side_hi": 320,
         "precision": FP32, "steps": 2},
        # the bar with the 3-D k-epsilon closure over a friction bed
        {"name": "bar_kepsilon_ragged_fp32", "kind": "run", "scene": "bar_ke", "M": 515, "N": 30, "K": 15,
         "precision": FP32, "steps": 4},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dt", "fluxes", "run", "run", "run", "run", "run", "run", "routines", "ensemble"])
    prec = rng.choice([FP32, FP32, FP64])
    if kind == "dt":
        return {"kind": kind, "M": _logint(rng, 48, 1024), "N": _logint(rng, 4, 512), "K": rng.randint(4, 24)}
    if kind == "fluxes":
        return {"kind": kind, "M": _logint(rng, 48, 512), "N": _logint(rng, 4, 256), "K": rng.randint(4, 24),
                "precision": prec}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 12), "sizes": rng.randint(8, 10 ** 6), "side_lo": 64,
                "side_hi": _logint(rng, 128, 320), "precision": FP32, "steps": rng.randint(1, 2)}
    scene = rng.choice(["channel", "bar", "beach", "basin", "flume", "bar_ke", "bar_les"])
    lo_m, hi_m, lo_n, hi_n, lo_k, hi_k = {
        "channel": (64, 1024, 4, 32, 4, 20), "bar": (96, 1024, 6, 64, 6, 32), "beach": (48, 512, 40, 512, 5, 12),
        "basin": (64, 512, 64, 512, 5, 24), "flume": (64, 1024, 4, 32, 5, 40), "bar_ke": (96, 768, 6, 48, 6, 20),
        "bar_les": (96, 512, 6, 32, 6, 20)}[scene]
    return {"kind": kind, "scene": scene, "M": _logint(rng, lo_m, hi_m), "N": _logint(rng, lo_n, hi_n),
            "K": rng.randint(lo_k, hi_k), "precision": prec, "steps": 1 if prec == FP64 else rng.randint(1, 4)}


# ------------------------------------------------------------- inputs
def _smooth(g, M, N, shortest, modes=16):
    """A seeded smooth random field [N][M] of unit size: cosine modes no shorter than ``shortest`` cells."""
    x, y = (np.arange(M) + 0.5)[None, :], (np.arange(N) + 0.5)[:, None]
    f = np.zeros((N, M))
    for _ in range(modes):
        th, lam = g.uniform(0.0, 2.0 * math.pi), shortest * g.uniform(1.0, 4.0)
        kx, ky, ph = 2 * math.pi * math.cos(th) / lam, 2 * math.pi * math.sin(th) / lam, g.uniform(0.0, 2 * math.pi)
        f += np.cos(kx * x + ph) * np.cos(ky * y) - np.sin(kx * x + ph) * np.sin(ky * y)
    return f / math.sqrt(modes)


def _basin(g, M, N, K, dx, precision):
    """Uneven bed of 5 to 200 m and a Gaussian hump at rest between walls, as the ensemble configuration has it."""
    f = _smooth(g, M, N, 40.0)
    f = (f - f.min()) / (f.max() - f.min())
    depth = 5.0 + 195.0 * f
    ci, cj = g.uniform(0.25, 0.75) * M, g.uniform(0.25, 0.75) * N
    amp = g.uniform(0.01, 0.1) * depth[int(cj), int(ci)]
    width = g.uniform(10.0, 40.0)
    ii, jj = np.arange(M)[None, :] + 0.5, np.arange(N)[:, None] + 0.5
    eta = amp * np.exp(-((ii - ci) ** 2 + (jj - cj) ** 2) / width ** 2)
    p = default_params(Mglob=M, Nglob=N, Kglob=K, dx=dx, dy=dx, dt_ini=0.4 * dx / math.sqrt(G * 200.0), dt_min=1e-8)
    p.precision = precision
    return p, depth.ravel(), eta.ravel(), None


def _scene(case, seed):
    """(params, depth, eta0, uvw0) of a run: its sizes from the case, its waves from the seed."""
    g = np.random.default_rng(int(seed))
    scene, M, N, K = case["scene"], case["M"], case["N"], case["K"]
    endless = dict(total_time=1.0e30, sim_steps=2 ** 31 - 1)
    if scene == "channel":
        out = scenarios.solitary_channel(M=M, N=N, K=K, amp=g.uniform(0.1, 0.2), x0=0.1 * M * g.uniform(0.2, 0.6),
                                         **endless)
    elif scene in ("bar", "bar_ke", "bar_les"):
        kw = dict(endless)
        if scene == "bar_ke":
            kw.update(viscous_flow=1, visc=1e-6, ivturb=10, ihturb=10, prod_type=3, bc_z0=5, ibot=1, cd0=0.006)
        elif scene == "bar_les":
            kw.update(viscous_flow=1, visc=1e-6, ivturb=20, ihturb=20, cvs=0.1)
        out = scenarios.submerged_bar(M=M, N=N, K=K, dx=25.6 / M, dy=0.05, **kw)
        out[0].amp_wave = g.uniform(0.008, 0.012)
        out = (out[0], out[1], 0.004 * _smooth(g, M, N, 0.1 * M).ravel(), None)
    elif scene == "beach":
        out = scenarios.landslide_beach(M=M, N=N, K=K, dx=1024.0 / M, **endless)
        p = out[0]
        p.slide_t, p.slide_x0, p.slide_y0 = g.uniform(6.0, 10.0), g.uniform(0.55, 0.62) * 1024.0, 0.5 * N * p.dy
        off_shore = np.clip((0.7 - (np.arange(M) + 0.5) / M) / 0.2, 0.0, 1.0)   # no wave at the dry beach yet
        out = (p, out[1], (0.2 * _smooth(g, M, N, 0.2 * M) * off_shore ** 2).ravel(), None)
    elif scene == "flume":
        out = scenarios.wave_flume("JON", M=M, N=N, K=K, hm0=0.03, tp=1.5, freq_min=0.4, freq_max=1.2, numfreq=24,
                                   wave_seed=int(g.integers(1, 10 ** 6)), **endless)
        out = (out[0], out[1], 0.004 * _smooth(g, M, N, 0.1 * M).ravel(), None)
    else:
        out = _basin(g, M, N, K, 4.0, FP64)
    p = out[0]
    p.precision = case["precision"]
    p.tol = 1e-12 if p.precision == FP64 else 1e-8
    return out


def _members(case):
    """Sizes of an ensemble's members: sides log-uniform, K of the configuration's four, dx log-uniform in 2 to 20 m."""
    r = random.Random(case["sizes"])
    return [(_logint(r, case["side_lo"], case["side_hi"]), _logint(r, case["side_lo"], case["side_hi"]),
             r.choice([5, 10, 15, 20]), math.exp(r.uniform(math.log(2.0), math.log(20.0))))
            for _ in range(case["members"])]


def _buffer(shape, name):
    """A pinned host buffer for one field, as a program that reads its fields every few steps keeps it."""
    shp, dtype = shape.of(getattr(F, name))
    return torch.empty(shp[::-1], dtype=torch.float64 if dtype == np.float64 else torch.int32, pin_memory=True).numpy()


def _dt_arrays(case, seed):
    """U, V, W, D and dsig of a host model, ghosts included, as [k][j][i]: waves over 1 m of water."""
    M, N, K = case["M"], case["N"], case["K"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    a = [0.3 * torch.randn(K + 4, N + 4, M + 4, dtype=torch.float64, device="cuda", generator=gen) for _ in range(3)]
    d = 1.0 + 0.1 * torch.rand(N + 4, M + 4, dtype=torch.float64, device="cuda", generator=gen)
    dsig = torch.full((K + 4,), float(np.float32(1.0) / np.float32(K)), dtype=torch.float64, device="cuda")
    return a + [d, dsig]


DT = dict(dx=0.1, dy=0.1, cfl=0.5, dt_old=1.0, dt_max=1.0)


def _flux_fields(case, seed):
    """Host fields of the state that the fluxes are taken of: waves over an uneven bed of about 10 m, ghosts included."""
    M, N, K = case["M"], case["N"], case["K"]
    g = np.random.default_rng(int(seed))
    depth = 10.0 + 2.0 * _smooth(g, M, N, 30.0)
    eta = 0.5 * _smooth(g, M + 4, N + 4, 20.0)
    lev = np.linspace(0.5, 1.0, K + 4)[:, None, None]
    vel = {n: _smooth(g, M + 4, N + 4, 20.0)[None] * lev * s + 0.01 * s * g.standard_normal((K + 4, N + 4, M + 4))
           for n, s in (("U", 1.0), ("V", 1.0), ("W", 0.2))}
    d = np.pad(depth, 2, mode="symmetric") + eta
    om = 0.05 * g.standard_normal((K + 5, N + 4, M + 4))
    return depth, dict(vel, ETA=eta, D=d, OMEGA=om, DU=d * vel["U"], DV=d * vel["V"], DW=d * vel["W"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dt":
        return {"kind": kind, "arrays": _dt_arrays(case, seed), "sizes": (case["M"], case["N"], case["K"]),
                "out": torch.zeros(1, dtype=torch.float64, device="cuda"), "lib": lib.load()}
    if kind == "fluxes":
        depth, fields = _flux_fields(case, seed)
        p = default_params(Mglob=case["M"], Nglob=case["N"], Kglob=case["K"], dx=2.0, dy=2.0)
        p.precision = case["precision"]
        s = lib.Scenario(p, depth.ravel())
        for n, a in fields.items():
            s.set(getattr(F, n), a)
        return {"kind": kind, "scenario": s, "fp32": p.precision == FP32,
                "out": {n: _buffer(s.shape, n) for n in FLUXES}}
    if kind == "ensemble":
        g = np.random.default_rng(int(seed))
        members = [lib.Scenario(*_basin(g, M, N, K, dx, case["precision"])) for M, N, K, dx in _members(case)]
        return {"kind": kind, "members": members, "ensemble": lib.Ensemble(members), "steps": case["steps"],
                "fp32": case["precision"] == FP32,
                "out": [{n: _buffer(m.shape, n) for n in STATE} for m in members]}
    p, depth, eta0, uvw0 = _scene(case, seed)
    s = lib.Scenario(p, depth, eta0, uvw0)
    names = STATE + (("MASK",) if case["scene"] == "beach" else ()) + (
        ("TKE", "EPS", "CMUVT") if case["scene"] == "bar_ke" else ())
    return {"kind": kind, "scenario": s, "steps": case["steps"], "fp32": p.precision == FP32,
            "sponge": bool(p.sponge_on), "out": {n: _buffer(s.shape, n) for n in names}}


# --------------------------------------------------------------- passes
def _fields(s, out, fp32):
    """The interior of the scenario's fields, read into the program's buffers; FP32 for the FP32+IR form."""
    got = {}
    for n, buf in out.items():
        f = getattr(F, n)
        a = torch.from_numpy(s.get(f, buf)[s.shape.interior(f)])
        got[n] = a.to(torch.float32) if fp32 and a.is_floating_point() else a
    return got


def run(state):
    kind = state["kind"]
    if kind == "dt":
        M, N, K = state["sizes"]
        st = state["lib"].nhw_estimate_dt_noalloc(
            *[a.data_ptr() for a in state["arrays"]], M, N, K, DT["dx"], DT["dy"], DT["cfl"], DT["dt_old"],
            DT["dt_max"], state["out"].data_ptr(), None)
        if st != lib.OK:
            raise RuntimeError(lib.last_error())
        return state["out"]
    if kind == "ensemble":
        state["ensemble"].step(state["steps"])
        return [_fields(m, out, state["fp32"]) for m, out in zip(state["members"], state["out"])]
    s = state["scenario"]
    if kind == "fluxes":
        s.fluxes()
    elif kind == "run":
        s.run(state["steps"])
    else:
        for _ in range(state["steps"]):
            s.estimate_dt()
            s.update_bathymetry()
            s.update_wave_bc()
            s.update_mask()
            s.update_vars()
            for stage in (1, 2, 3):
                s.source_terms()
                s.fluxes()
                s.eval_duvw(stage)
                if state["sponge"]:
                    s.sponge_damping()
                s.eval_turb(stage)
    return _fields(s, state["out"], state["fp32"])


# ----------------------------------------------------------------- work
def work(case):
    """Bytes: a step reads and writes its state once (U, V, W, DU, DV, DW in the form's precision, P in FP64) and a
    pass hands its output fields to the host once.  Flops: per cell and stage about 400 for reconstruction, fluxes,
    update and projection, and 60 for one application of the pressure operator and of a smoother."""
    kind = case["kind"]
    if kind == "dt":
        n, n2 = case["M"] * case["N"] * case["K"], case["M"] * case["N"]
        return {"bytes": 24 * n + 8 * n2 + 8, "flops": 12 * n}
    sizes = [m[:3] for m in _members(case)] if kind == "ensemble" else [(case["M"], case["N"], case["K"])]
    n, n2 = sum(a * b * c for a, b, c in sizes), sum(a * b for a, b, _ in sizes)
    s = 4 if case["precision"] == FP32 else 8
    if kind == "fluxes":
        return {"bytes": n * (6 * s + s) + 8 * n2 + n * 11 * 8, "flops": 400 * n}
    per_step = n * (2 * 6 * s + 16) + 16 * n2
    return {"bytes": case["steps"] * per_step + 8 * (4 * n + n2), "flops": case["steps"] * 3 * 460 * n}


# ---------------------------------------------------------------- exact
def _slope(a, d0, d1, dim):
    """Van Leer limited slope of ``a`` along ``dim`` at all but the two end cells; d0, d1 the spacings below and above."""
    n = a.shape[dim]
    t1 = (a.narrow(dim, 2, n - 2) - a.narrow(dim, 1, n - 2)) / d1
    t2 = (a.narrow(dim, 1, n - 2) - a.narrow(dim, 0, n - 2)) / d0
    s = t1.abs() + t2.abs()
    return torch.where(s < 1e-16, torch.zeros_like(s), (t1 * t2.abs() + t1.abs() * t2) / s.clamp_min(1e-300))


def _hll(sl, sr, fl, fr, du):
    mid = (sr * fl - sl * fr + sl * sr * du) / (sr - sl)
    return torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, mid))


def _lateral(v, normal, eta, depth, h, dim):
    """HLL fluxes through the faces across ``dim`` (-1: x, -2: y) of an all-wet walled basin, in 64 bits: mass, then
    momentum in x, y, z.  v: U, V, W, DU, DV, DW with one ghost cell more than the faces need on both sides."""
    def sides(a):
        n = a.shape[dim]
        half = 0.5 * h * _slope(a, h, h, dim)
        c = a.narrow(dim, 1, n - 2)
        m = n - 3
        return (c + half).narrow(dim, 0, m), (c - half).narrow(dim, 1, m)
    eL, eR = sides(eta)
    n = depth.shape[dim]
    hf = 0.5 * (depth.narrow(dim, 1, n - 3) + depth.narrow(dim, 2, n - 3))
    dL, dR = (eL + hf).clamp_min(0.01), (eR + hf).clamp_min(0.01)
    L, R = zip(*[sides(a) for a in v])
    uL, uR = L[normal], R[normal]
    cL, cR = (G * dL).sqrt(), (G * dR).sqrt()
    cS, uS = 0.5 * (cL + cR) + 0.25 * (uL - uR), 0.5 * (uL + uR) + cL - cR
    sl, sr = torch.minimum(uL - cL, uS - cS), torch.maximum(uR + cR, uS + cS)
    pL, pR = [0.5 * G * (e * e + 2.0 * e * hf) for e in (eL, eR)]
    out = [_hll(sl, sr, L[3 + normal], R[3 + normal], dR - dL)]
    for q in range(3):
        fl = L[3 + q] * uL + pL if q == normal else dL * uL * L[q]
        fr = R[3 + q] * uR + pR if q == normal else dR * uR * R[q]
        out.append(_hll(sl, sr, fl, fr, R[3 + q] - L[3 + q]))
    walls = out[0].shape[dim] - 1
    for q, a in enumerate(out):   # closed walls: the hydrostatic pressure alone
        for at, wall in ((0, pR), (walls, pL)):
            a.select(dim, at).copy_(wall.select(dim, at) if q == 1 + normal else torch.zeros_like(a.select(dim, at)))
    return out


def _exact_fluxes(case, seed):
    depth, fields = _flux_fields(case, seed)
    M, N, K = case["M"], case["N"], case["K"]
    t = {n: torch.from_numpy(a) for n, a in fields.items()}
    hc = torch.from_numpy(np.pad(depth, 2, mode="symmetric"))
    cells = [t[n][2:2 + K] for n in ("U", "V", "W", "DU", "DV", "DW")]
    x = _lateral([a[:, 2:2 + N] for a in cells], 0, t["ETA"][2:2 + N], hc[2:2 + N], 2.0, -1)
    y = _lateral([a[:, :, 2:2 + M] for a in cells], 1, t["ETA"][:, 2:2 + M], hc[:, 2:2 + M], 2.0, -2)
    ds, om = float(np.float32(1.0) / np.float32(K)), t["OMEGA"][2:3 + K, 2:2 + N, 2:2 + M]
    out = dict(zip(FLUXES[:8], x + y))
    for n, name in (("U", "FZ"), ("V", "GZ"), ("W", "HZ")):
        a = t[n][:, 2:2 + N, 2:2 + M]
        half = 0.5 * ds * _slope(a, ds, ds, 0)
        lo, hi = (a[1:-1] + half)[:K + 1], (a[1:-1] - half)[1:K + 2]
        f = 0.5 * (om * (lo + hi) - om.abs() * (hi - lo))
        f[0], f[K] = 0.0, 0.0
        out[name] = f
    return {n: out[n] for n in FLUXES}


def exact(case, seed):
    """What ``run`` returns, in 64 bits, where it has a closed value: the time step and the fluxes.  A whole step has
    none: its pressure is whatever the iterative solve stops at within the tolerance."""
    if case["kind"] == "dt":
        u, v, w, d, dsig = _dt_arrays(case, seed)
        c = slice(2, -2)
        u, v, w, d = u[c, c, c], v[c, c, c], w[c, c, c], d[c, c]
        root = (G * d).sqrt()[None]
        bound = min(float((DT["dx"] / (u.abs() + root)).min()), float((DT["dy"] / (v.abs() + root)).min()),
                    float((dsig[c][:, None, None] * d[None] / w.abs().clamp_min(1e-16)).min()))
        return torch.tensor([min(float(np.float32(1.05)) * DT["dt_old"], DT["cfl"] * bound, DT["dt_max"])],
                            dtype=torch.float64)
    if case["kind"] == "fluxes":
        return _exact_fluxes(case, seed)
    return None
