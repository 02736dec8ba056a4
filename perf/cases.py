"""The workloads this engine is timed on: what its users run, through its public entry points.

A case is a bed (or a batch of beds, or the network of the learned warm
start), its precision and the number of time steps of one pass.  prepare()
makes the bed from the seed and commits it to an engine handle, as a program
does once; run() is one pass: ``steps`` time steps and the read of the
particle state into page-locked host arrays, which is what the time loop of
a program does between two outputs.  State fields come back in the precision
the build holds them in: the FP32 build's are stored as float32 (its DEM
state too, as a plot or restart file stores it), positions and the FP64
build's fields as float64.
"""
import ctypes as C
import math

import numpy as np
import torch

from fluidized_bed_master_b200 import beds
from fluidized_bed_master_b200.engine import Engine, lib
from fluidized_bed_master_b200.params import (DEM, PPE_PCG, PRECOND_JACOBI, PRECOND_TWO_LEVEL, SPH, WARM_PREVIOUS,
                                              WARM_PROJECT)

POSITIONS = ("x", "y", "z")
SPH_OUT = ("ux", "uy", "uz", "rho", "pres", "temp", "DEMpor", "ftotalz", "fpz")
DEM_OUT = ("x", "y", "z", "ux", "uy", "uz", "wx", "wy", "wz", "temp", "ftotalx", "ftotalz")
W_OUT = ("x", "y", "ux", "uy", "rho", "pres", "drho")
# the mutable state that a host program which owns the particles hands over each step
SPH_STATE = ("ux", "uy", "uz", "m", "rho", "pres", "temp", "dDEMpor", "flt_s")
DEM_STATE = ("x", "y", "z", "ux", "uy", "uz", "wx", "wy", "wz", "temp", "Fdx_df", "Fdy_df", "Fdz_df", "Q_sd")


def listed():
    return [
        # a coarse spouted bed (the smoke test's size): launches and latency
        {"name": "spouted_small", "kind": "spouted", "dx": 2.0e-3, "r_dem": 1.0e-3, "n_dem": 300, "spacing": 2.1,
         "precision": 0, "steps": 40},
        # the reference's own scenario: gas-spouted bed in its cylinder and cone, Wendland C6
        {"name": "spouted", "kind": "spouted", "dx": 0.5e-3, "r_dem": 0.5e-3, "n_dem": 4580, "spacing": 2.1,
         "precision": 0, "steps": 20},
        # the benchmark bed: 301,760 SPH + 20,000 DEM with heat transfer
        {"name": "box", "kind": "box", "n_fluid": 200_000, "n_dem": 20_000, "lx": 0.1, "precision": 0, "heat": 1,
         "steps": 20},
        # the same in double precision, for validation runs
        {"name": "box_fp64", "kind": "box", "n_fluid": 200_000, "n_dem": 20_000, "lx": 0.1, "precision": 1, "heat": 1,
         "steps": 10},
        # the engine as the step operator of a host program that owns the particles: whole state in and out per step
        {"name": "box_exchange", "kind": "exchange", "n_fluid": 200_000, "n_dem": 20_000, "lx": 0.1, "precision": 0,
         "heat": 1, "steps": 4},
        # the bed ten times as wide: 2.8 M SPH + 200,000 DEM
        {"name": "scaled", "kind": "box", "n_fluid": 2_000_000, "n_dem": 200_000, "lx": 1.0, "precision": 0, "heat": 1,
         "steps": 8},
        # the bed with the pressure equation solved to 1e-6: two-level PCG, projected start
        {"name": "box_pcg", "kind": "pcg", "n_fluid": 200_000, "n_dem": 20_000, "lx": 0.1, "precision": 0, "heat": 1,
         "two_level": 1, "project": 2, "steps": 5},
        # the 3-D ISPH column (dx 4 mm, 332,416 particles), Jacobi-PCG to 1e-6
        {"name": "column", "kind": "column", "dx": 4.0e-3, "precision": 0, "two_level": 0, "steps": 4},
        # 64 uneven 2-D SPH-DEM beds served from one handle
        {"name": "bed2d_batch", "kind": "bed2d_batch", "n_beds": 64, "n_min": 2_000, "n_max": 50_000, "sizes": 0,
         "precision": 0, "steps": 12},
        # the 2-D WCSPH dam break (14,978 particles)
        {"name": "dam2d", "kind": "dam2d", "dx": 5.0e-3, "precision": 0, "kgc": 0, "delta": 0, "xsph": 0, "steps": 40},
        # 64 uneven dam breaks in one handle
        {"name": "dam2d_batch", "kind": "dam2d_batch", "n_beds": 64, "n_min": 2_000, "n_max": 50_000, "sizes": 0,
         "precision": 0, "steps": 10},
        # one training pass of the learned warm start's network over the scaled bed's rows
        {"name": "mlp", "kind": "mlp", "rows": 2_827_520},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["spouted", "box", "box", "exchange", "pcg", "column", "bed2d_batch", "dam2d", "dam2d_batch",
                       "mlp"])
    if kind == "spouted":
        r = rng.choice([0.5e-3, 0.75e-3, 1.0e-3])
        return {"kind": kind, "dx": round(_log(rng, 0.5e-3, 2.0e-3), 6), "r_dem": r, "n_dem": int(_log(rng, 50, 4580)),
                "spacing": round(rng.uniform(2.05, 2.3), 3), "precision": int(rng.random() < 0.25), "steps": 20}
    if kind in ("box", "exchange", "pcg"):
        n = int(_log(rng, 5_000, 400_000 if kind == "box" else 250_000)) | 1
        c = {"kind": kind, "n_fluid": n, "n_dem": int(n * rng.uniform(0.02, 0.1)), "lx": rng.choice([0.05, 0.1, 0.2]),
             "precision": int(rng.random() < 0.25) if kind == "box" else 0, "heat": int(rng.random() < 0.75),
             "steps": {"box": 10, "exchange": 4, "pcg": 3}[kind]}
        if kind == "pcg":
            c.update(two_level=int(rng.random() < 0.7), project=rng.choice([0, 2, 4]))
        return c
    if kind == "column":
        return {"kind": kind, "dx": round(_log(rng, 4.0e-3, 1.2e-2), 6), "precision": 0,
                "two_level": int(rng.random() < 0.5), "steps": 4}
    if kind == "bed2d_batch":
        return {"kind": kind, "n_beds": int(_log(rng, 1, 65)), "n_min": 2_000, "n_max": rng.choice([10_000, 50_000]),
                "sizes": rng.randrange(1000), "precision": int(rng.random() < 0.2), "steps": 10}
    if kind == "dam2d":
        return {"kind": kind, "dx": round(_log(rng, 2.5e-3, 1.2e-2), 6), "precision": int(rng.random() < 0.25),
                "kgc": int(rng.random() < 0.3), "delta": rng.choice([0, 0, 1, 2]), "xsph": int(rng.random() < 0.3),
                "steps": 20}
    if kind == "dam2d_batch":
        return {"kind": kind, "n_beds": int(_log(rng, 2, 65)), "n_min": 2_000, "n_max": rng.choice([10_000, 50_000]),
                "sizes": rng.randrange(1000), "precision": 0, "steps": 10}
    return {"kind": "mlp", "rows": int(_log(rng, 1_000, 2_827_520))}


# ---- beds ------------------------------------------------------------------
def _bed(case, seed):
    """(params, sph, dem, rows of a 2-D batch) of a case."""
    k = case["kind"]
    rows = None
    if k == "spouted":
        p, sph, dem = beds.spouted_bed(dx=case["dx"], r_dem=case["r_dem"], n_dem=case["n_dem"],
                                       spacing=case["spacing"], u_dem=0.05, seed=seed)
    elif k in ("box", "exchange", "pcg"):
        p, sph, dem = beds.box_bed(n_fluid=case["n_fluid"], n_dem=case["n_dem"], lx=case["lx"], seed=seed)
        p.con_solve = case["heat"]
    elif k == "column":
        p, sph, dem = beds.isph_column(dx=case["dx"], seed=seed)
    elif k == "bed2d_batch":
        # "sizes" draws the beds' particle counts and inlets, the seed their particles' positions and temperatures
        p, sph, dem, rows, _ = beds.bed2d_batch(n_beds=case["n_beds"], n_min=case["n_min"], n_max=case["n_max"],
                                                seed=case["sizes"])
        rng = np.random.default_rng(seed)
        n = len(sph["x"])
        sph["x"] = sph["x"] + rng.uniform(-1e-5, 1e-5, n)
        sph["z"] = sph["z"] + rng.uniform(-1e-5, 1e-5, n)
        sph["temp"] = sph["temp"] + rng.uniform(-1.0, 1.0, n)
    else:
        p, sph, dem = beds.dam_break_2d(dx=case["dx"], seed=seed)
        p.kgc_solve, p.delSPH_solve, p.xsph_solve = case["kgc"], case["delta"], case["xsph"]
    p.precision = case["precision"]
    if k in ("pcg", "column"):
        p.ppe_mode = PPE_PCG
        p.ppe_tol = 1.0e-6
        p.ppe_max_iter = 2000
        p.kgc_solve = 0          # the CG needs the uncorrected (symmetric) operator
        p.ppe_precond = PRECOND_TWO_LEVEL if case["two_level"] else PRECOND_JACOBI
        hist = case.get("project", 0)
        p.warm_start = WARM_PROJECT if hist else WARM_PREVIOUS
        p.warm_hist = hist or 8
    return p, sph, dem, rows


def _pinned(names, n):
    """A page-locked [field, particle] block and its rows by name."""
    t = torch.empty((len(names), n), dtype=torch.float64, pin_memory=True)
    a = t.numpy()
    return t, {f: a[k] for k, f in enumerate(names)}


class _Read:
    """The read of one particle set: page-locked double arrays, and the float32 copy that a program stores."""

    def __init__(self, which, names, n, single):
        self.which, self.names = which, names
        self.block, self.rows = _pinned(names, n)
        self.n_pos = sum(f in POSITIONS for f in names) if single else len(names)
        self.f32 = torch.empty((len(names) - self.n_pos, n), dtype=torch.float32)

    def __call__(self, eng):
        eng.get_fields(self.which, self.rows)
        self.f32.copy_(self.block[self.n_pos:])
        out = {f: self.block[k] for k, f in enumerate(self.names[:self.n_pos])}
        out.update({f: self.f32[k] for k, f in enumerate(self.names[self.n_pos:])})
        return out


def prepare(case, seed):
    k = case["kind"]
    if k == "mlp":
        return _prepare_mlp(case, seed)
    if k == "dam2d_batch":
        p, parts = beds.dam_break_batch(n_beds=case["n_beds"], n_min=case["n_min"], n_max=case["n_max"],
                                        seed=case["sizes"])
        rng = np.random.default_rng(seed)
        for b in parts:
            b["x"] = b["x"] + rng.uniform(-2e-5, 2e-5, len(b["x"]))
            b["y"] = b["y"] + rng.uniform(-2e-5, 2e-5, len(b["x"]))
        p.precision = case["precision"]
        eng = Engine.batch(p, parts)
    else:
        p, sph, dem, rows = _bed(case, seed)
        eng = Engine(p, sph, dem, beds=rows)
    single = case["precision"] == 0
    out_s = W_OUT if k in ("dam2d", "dam2d_batch") else SPH_OUT
    s = {"kind": k, "eng": eng, "steps": case["steps"], "read": [_Read(SPH, out_s, eng.ns, single)]}
    if eng.nd:
        s["read"].append(_Read(DEM, DEM_OUT, eng.nd, single))
    if k not in ("dam2d", "dam2d_batch"):
        s["start"] = _host_state(eng)
        if k == "exchange":
            s["host"] = _host_state(eng)
    return s


def _host_state(eng):
    """The engine's mutable state in page-locked host arrays: fields of both sets, contact history."""
    sets, history = [], None
    for which, names, n in ((SPH, SPH_STATE, eng.ns), (DEM, DEM_STATE, eng.nd)):
        if n:
            keep, rows = _pinned(names, n)
            eng.get_fields(which, rows)
            sets.append((which, rows, keep))
    if eng.nd:
        ids = torch.empty((eng.nd, 16), dtype=torch.int32, pin_memory=True).numpy()
        springs = torch.empty((eng.nd, 16, 3), dtype=torch.float64, pin_memory=True).numpy()
        history = eng.history(out=(ids, springs))
    return sets, history


def _set_state(eng, host):
    for which, rows, _keep in host[0]:
        eng.set_fields(which, rows)
    if host[1] is not None:
        eng.set_history(*host[1])


def run(state):
    k = state["kind"]
    if k == "mlp":
        return _run_mlp(state)
    eng = state["eng"]
    if "start" in state:
        _set_state(eng, state["start"])
    if k == "exchange":
        # every step: one step, state and contact history to the host, and back for the next
        host = state["host"]
        for q in range(state["steps"]):
            if q:
                _set_state(eng, host)
            eng.step(1)
            for which, rows, _keep in host[0]:
                eng.get_fields(which, rows)
            eng.history(out=host[1])
    else:
        eng.step(state["steps"])
    return {"dem" if r.which == DEM else "sph": r(eng) for r in state["read"]}


# ---- the network of the learned warm start -----------------------------------
N_IN, N_H = 16, 64


def _mlp_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    n = case["rows"]
    return (torch.randn(n, N_IN, generator=g).to(torch.bfloat16),
            0.2 * torch.randn(N_H * N_IN + N_H + N_H * N_H + N_H + N_H + 1, generator=g),
            torch.randn(n, generator=g), (torch.rand(n, generator=g) > 0.2).float())


def _prepare_mlp(case, seed):
    L = lib()
    L.sphdem_mlp_forward.argtypes = [C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    L.sphdem_mlp_grad.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_double, C.c_void_p,
                                  C.c_void_p]
    feat, params, target, weight = (t.cuda() for t in _mlp_inputs(case, seed))
    n = case["rows"]
    return {"kind": "mlp", "lib": L, "n": n, "feat": feat, "params": params, "target": target, "weight": weight,
            "weight_sum": float(weight.sum()), "out": torch.empty(n, dtype=torch.float32, device="cuda"),
            "grad": torch.empty(params.numel() + 2, dtype=torch.float32, device="cuda")}


def _run_mlp(s):
    st = torch.cuda.current_stream().cuda_stream
    r = s["lib"].sphdem_mlp_forward(s["feat"].data_ptr(), s["n"], s["params"].data_ptr(), s["out"].data_ptr(), st)
    r |= s["lib"].sphdem_mlp_grad(s["feat"].data_ptr(), s["target"].data_ptr(), s["weight"].data_ptr(), s["n"],
                                  s["params"].data_ptr(), s["weight_sum"], s["grad"].data_ptr(), st)
    if r:
        raise RuntimeError(f"network entry returned {r}")
    return {"out": s["out"], "grad": s["grad"]}


# ---- what a pass cannot do without ---------------------------------------------
def work(case):
    """Bytes: every step reads and writes each particle's state once (positions and radii FP64, DEM state FP64, SPH
    fields in the build's precision) and the pass writes its outputs once.  Operations: the pair sums of a step,
    counted by hand from the equations (pressure, viscous, heat, gradient-correction, Poisson and smoothing sums over
    the neighbours; contact and drag per sphere)."""
    k = case["kind"]
    if k == "mlp":
        n = case["rows"]
        return {"bytes": n * (2 * N_IN * 2 + 4 + 8), "flops": n * (10_368 + 29_120)}
    r = 8 if case["precision"] else 4
    nd = 0
    nbr, per_pair = 76, 190
    if k == "spouted":
        ns = int(109_098 * (0.5e-3 / case["dx"]) ** 3)
        nd, nbr = case["n_dem"], 110
    elif k in ("box", "exchange", "pcg"):
        ns, nd = int(case["n_fluid"] * (1.5 if case["lx"] <= 0.1 else 1.4)), case["n_dem"]
    elif k == "column":
        ns, per_pair = int(332_416 * (4.0e-3 / case["dx"]) ** 3), 120
    elif k in ("bed2d_batch", "dam2d_batch"):
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        ns, nbr = int(case["n_beds"] * mean * 1.05), 21
        nd = int(0.09 * ns) if k == "bed2d_batch" else 0
    else:
        ns, nbr = int(14_978 * (5.0e-3 / case["dx"]) ** 2), 21
    if k in ("dam2d", "dam2d_batch"):
        state, per_pair = 2 * (6 * 8 + 5 * r), 70
    else:
        state = 4 * 8 + 2 * 10 * r   # SPH positions do not change in these steps
    step = ns * state + nd * 2 * 22 * 8
    out = (ns * 9 + nd * 12) * 8
    flops = ns * nbr * per_pair + nd * 4_000
    n = case["steps"]
    if k not in ("dam2d", "dam2d_batch"):
        out += (2 * n if k == "exchange" else 1) * (ns * 9 * 8 + nd * (14 * 8 + 16 * 28))
    return {"bytes": n * step + out, "flops": n * flops}


# ---- 64-bit values, without the engine -------------------------------------------
def exact(case, seed):
    """The network's outputs and a single dam break's fields in 64 bits with torch and numpy.  The other beds have no
    such value here: a step of the coupled model in plain numpy takes longer than the comparison may."""
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    if case["kind"] == "dam2d" and not (case["kgc"] or case["delta"] or case["xsph"]) and case["dx"] > 3.0e-3:
        return {"sph": _exact_dam2d(case, seed)}
    return None


def _exact_mlp(case, seed):
    feat, params, target, weight = _mlp_inputs(case, seed)
    rnd = lambda t: t.float().to(torch.bfloat16).double()   # noqa: E731  operands of the matrix units are BF16
    p = params.double()
    cut = np.cumsum([N_H * N_IN, N_H, N_H * N_H, N_H, N_H])
    W1, b1, W2, b2, w3, b3 = (p[a:b] for a, b in zip([0, *cut], [*cut, len(p)]))
    W1, W2, w3 = rnd(W1).view(N_H, N_IN), rnd(W2).view(N_H, N_H), rnd(w3)
    wsum, out, g = float(weight.sum()), [], torch.zeros(len(p) + 2, dtype=torch.float64)
    for a in range(0, case["rows"], 1 << 18):
        x, t, w = feat[a:a + (1 << 18)].double(), target[a:a + (1 << 18)].double(), weight[a:a + (1 << 18)].double()
        z1 = x @ W1.T + b1
        h1 = rnd(z1.clamp(min=0))
        h2 = (h1 @ W2.T + b2).clamp(min=0)
        y = h2 @ w3 + b3
        e = y - t
        g3 = 2.0 * w * e / wsum
        d2 = rnd(torch.where(h2 > 0, g3[:, None] * w3, 0.0))
        d1 = rnd(torch.where(z1 > 0, d2 @ W2, 0.0))
        g += torch.cat([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0),
                        (g3[:, None] * h2).sum(0), g3.sum()[None], (w * e * e).sum()[None], w.sum()[None]])
        out.append(y)
    return {"out": torch.cat(out), "grad": g}


def _exact_dam2d(case, seed):
    """Predictor, cell order, neighbours (distance + 1e-20 < kappa h), continuity, Tait pressure, pressure, viscous
    and artificial-viscosity forces, corrector; particles in the cell order of the last step."""
    p, s, _ = beds.dam_break_2d(dx=case["dx"], seed=seed)
    st = {f: np.array(s[f], dtype=np.float64) for f in ("x", "y", "ux", "uy", "m", "rho", "h")}
    n = len(st["x"])
    st["fluid"] = (np.asarray(s["p_type"]) > 0).astype(np.float64)
    for f in ("fx", "fy", "drho", "pres"):
        st[f] = np.zeros(n)
    lo = np.array([st["x"][:-1].min(), st["y"][:-1].min()])
    hi = np.array([st["x"][:-1].max(), st["y"][:-1].max()])
    margin = p.margin
    lo[0] -= (hi[0] - lo[0]) * margin[0]
    hi[0] += (hi[0] - lo[0]) * margin[1]
    lo[1] -= (hi[1] - lo[1]) * margin[2]
    hi[1] += (hi[1] - lo[1]) * margin[3]
    cell = 1.1 * p.kappa * st["h"][0]
    NI, NJ = int((hi[0] - lo[0]) / cell) + 1, int((hi[1] - lo[1]) / cell) + 1

    def coords():
        i = np.clip(np.minimum(np.floor((st["x"] - lo[0]) / (hi[0] - lo[0]) * NI), NI - 1), 0, None).astype(np.int64)
        j = np.clip(np.minimum(np.floor((st["y"] - lo[1]) / (hi[1] - lo[1]) * NJ), NJ - 1), 0, None).astype(np.int64)
        return i, j

    def sort_cells():
        i, j = coords()
        order = np.argsort(i + NI * j, kind="stable")
        for f in st:
            st[f] = st[f][order]

    sort_cells()   # the order at commit
    B = p.soundspeed ** 2 * 1.186 / p.gamma
    for _ in range(case["steps"]):
        f, hdt = st["fluid"], 0.5 * p.dt
        st.update(x0=st["x"], y0=st["y"], ux0=st["ux"], uy0=st["uy"], rho0=st["rho"])
        st["x"], st["y"] = st["x"] + st["ux"] * hdt * f, st["y"] + st["uy"] * hdt * f
        st["ux"], st["uy"] = st["ux"] + st["fx"] * hdt, st["uy"] + st["fy"] * hdt
        st["rho"] = st["rho"] + st["drho"] * hdt * f
        sort_cells()
        # candidate pairs: three runs of three cells each
        ci, cj = coords()
        start = np.searchsorted(ci + NI * cj, np.arange(NI * NJ + 1))
        I, J = [], []
        for dj in (-1, 0, 1):
            ok = (cj + dj >= 0) & (cj + dj < NJ)
            row = np.flatnonzero(ok)
            base = NI * (cj[row] + dj)
            a, b = start[base + np.maximum(ci[row] - 1, 0)], start[base + np.minimum(ci[row] + 1, NI - 1) + 1]
            cnt = b - a
            I.append(np.repeat(row, cnt))
            J.append(np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(a, cnt))
        I, J = np.concatenate(I), np.concatenate(J)
        dx, dy = st["x"][I] - st["x"][J], st["y"][I] - st["y"][J]
        r = np.sqrt(dx * dx + dy * dy) + 1e-20
        ok = r < p.kappa * st["h"][I]
        I, J, dx, dy, r = I[ok], J[ok], dx[ok], dy[ok], r[ok]
        h = st["h"][I]
        q = 0.5 * r / h
        dw = np.where(q < 1, 2.228169203286535 / (4 * h * h) / (2 * h) * (-20 * q * (1 - q) ** 3), 0.0)
        gx, gy = dw * dx / r, dw * dy / r
        m, rho, f = st["m"], st["rho"], st["fluid"]
        add = lambda v: np.bincount(I, v, minlength=n)   # noqa: E731
        ux, uy = st["ux"] * f, st["uy"] * f
        rho_ref = m / (st["h"] / 1.6) ** 2
        tm = m[J] * rho[I] / rho[J]
        st["drho"] = add((ux[I] - ux[J]) * tm * gx + (uy[I] - uy[J]) * tm * gy) * rho / rho_ref
        st["pres"] = B * ((rho / rho_ref) ** p.gamma - 1.0)
        pr, vx, vy = st["pres"], st["ux"][I] - st["ux"][J], st["uy"][I] - st["uy"][J]
        cp = -m[J] * (pr[I] + pr[J]) / (rho[I] * rho[J])
        cv = (dx * gx + dy * gy) * 4 * m[J] / (rho[I] * rho[J]) * (p.mu_gas / 2) / (r * r)
        u = vx * dx + vy * dy
        hij = 0.5 * (st["h"][I] + st["h"][J])
        phi = hij * u / (r * r + 0.01 * hij * hij)
        pij = m[I] * phi * (-p.art_visc_alpha * p.soundspeed + p.art_visc_beta * phi) / (rho[I] + rho[J]) * 0.5
        pij = np.where(u < 0, pij, 0.0) * p.fva_solve
        st["fx"] = add(cp * gx + cv * vx - pij * gx)
        st["fy"] = add(cp * gy + cv * vy - pij * gy) - p.g_sph
        ux, uy = st["ux0"] + st["fx"] * p.dt * f, st["uy0"] + st["fy"] * p.dt * f
        fast = ux * ux + uy * uy >= p.u_limit ** 2
        st["ux"], st["uy"] = np.where(fast, st["ux0"], ux), np.where(fast, st["uy0"], uy)
        st["x"], st["y"] = st["x0"] + st["ux"] * p.dt * f, st["y0"] + st["uy"] * p.dt * f
        st["rho"] = np.where(f > 0, st["rho0"] + st["drho"] * p.dt, st["rho"])
    return {f: torch.from_numpy(st[f]) for f in W_OUT}
