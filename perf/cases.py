"""Workloads of this package and what they compute, for timing and comparing builds.

listed() names the workloads, draw(rng) makes others of the same ranges,
prepare(case, seed) makes the inputs and whatever a caller keeps between calls
(a loaded context, a batch), run(state) is one call of the public entry points
and returns its outputs whole, work(case) counts what the call cannot do
without, and exact(case, seed) states the outputs in 64 bits with torch and
numpy alone.

The kinds of call:
  patch     run_stage2 of an in-memory patch: preparation, random-phase
            histogram, upload, loop to convergence, every pm1 variable back
  loop      a loaded context's gamma loop from its first iteration to
            convergence, the per-PS results back
  batch     many loaded patches run together (batch.Batch)
  gradient  coherence of every PS and its gradients (autograd.coherence)
  stage3    the stage-3 re-estimate of the coherent PS of a patch that has
            just run stage 2, results kept on the device
  histogram the random-phase coherence histogram a patch's preparation needs
  topofit   the kernel registry's topofit over rows in host memory
  coherence the registry's topofit of one baseline vector, coherence only
"""
import math
import re
from pathlib import Path

import numpy as np
import torch

from pystamps_b200 import autograd, batch, kernels, stage2, stage3

DEV = torch.device("cuda", 0)
LAMBDA, RHO, CELL = 0.0555, 830_000.0, 50.0
SUMMARY = ("K_ps", "C_ps", "coh_ps", "N_opt", "Nr")
PM1 = ("K_ps", "C_ps", "coh_ps", "N_opt", "ph_res", "ph_patch", "ph_grid", "ph_weight", "coh_ps_save", "Nr")
NEAR_MAX = 2.0e-4


def listed():
    return [
        # the smallest whole call: a short stack over a small crop
        {"name": "patch-small", "kind": "patch", "n_ps": 5_000, "n_ifg": 18, "cells": 33, "trials": 61, "n_rand": 300_000},
        # a burst-sized patch as the reference's own benchmark has it; short kernels, launches count
        {"name": "loop-small", "kind": "loop", "n_ps": 20_000, "n_ifg": 20, "cells": 64, "trials": 81,
         "precision": "fp32", "weighting": "P-square", "row_variant": True},
        # an ordinary patch
        {"name": "loop-ordinary", "kind": "loop", "n_ps": 250_000, "n_ifg": 60, "cells": 128, "trials": 161,
         "precision": "fp32", "weighting": "P-square", "row_variant": True},
        # the largest: a dense patch with a long stack
        {"name": "loop-full-scale", "kind": "loop", "n_ps": 2_000_000, "n_ifg": 150, "cells": 256, "trials": 161,
         "precision": "fp32", "weighting": "P-square", "row_variant": True},
        # the plain FP64 path that results are checked with
        {"name": "loop-fp64", "kind": "loop", "n_ps": 100_000, "n_ifg": 40, "cells": 96, "trials": 121,
         "precision": "fp64", "weighting": "P-square", "row_variant": True},
        # SNR weighting, one baseline vector for all rows, ragged sizes
        {"name": "loop-snr", "kind": "loop", "n_ps": 61_803, "n_ifg": 33, "cells": 77, "trials": 121,
         "precision": "fp32", "weighting": "SNR", "row_variant": False},
        # a scene's uneven patches together
        {"name": "batch-uneven", "kind": "batch", "patches": 12, "ps_lo": 5_000, "ps_hi": 200_000, "trials": 161},
        # CLAP calibration: forward and backward
        {"name": "gradient", "kind": "gradient", "n_ps": 100_000, "n_ifg": 40, "cells": 96, "trials": 121},
        # PS selection after stage 2
        {"name": "stage3", "kind": "stage3", "n_ps": 250_000, "n_ifg": 60, "cells": 128, "trials": 161},
        # setup of a patch: the reference's 300,000 random rows
        {"name": "histogram", "kind": "histogram", "n_rand": 300_000, "n_ifg": 60, "trials": 161},
        # registry kernels: complex64 rows with their own baselines, some pixels missing
        {"name": "topofit-rows", "kind": "topofit", "n_ps": 20_000, "n_ifg": 40, "trials": 121, "single": True},
        # registry kernels: complex128 random-phase rows, one baseline vector
        {"name": "coherence-rows", "kind": "coherence", "n_ps": 30_000, "n_ifg": 30, "trials": 81},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    trials = 2 * rng.randint(20, 87) + 1
    kind = rng.choice(["patch", "loop", "loop", "loop", "batch", "gradient", "stage3", "histogram", "topofit", "coherence"])
    if kind == "batch":
        return {"kind": kind, "patches": rng.randint(3, 12), "ps_lo": log(2_000, 8_000), "ps_hi": log(40_000, 160_000),
                "trials": trials}
    if kind == "histogram":
        return {"kind": kind, "n_rand": log(30_000, 300_000), "n_ifg": rng.randint(8, 60), "trials": trials}
    if kind in ("topofit", "coherence"):
        c = {"kind": kind, "n_ps": log(300, 25_000), "n_ifg": rng.randint(9, 60), "trials": trials}
        return dict(c, single=rng.random() < 0.7) if kind == "topofit" else c
    n_ifg = log(10, 150)
    top = {"patch": 40_000, "loop": 1_200_000, "gradient": 150_000, "stage3": 300_000}[kind]
    n_ps = log(3_000, top)
    n_ps = max(2_000, min(n_ps, {"patch": 2_000_000, "gradient": 6_000_000}.get(kind, 60_000_000) // n_ifg))
    c = {"kind": kind, "n_ps": n_ps, "n_ifg": n_ifg, "cells": max(24, int(math.sqrt(n_ps / rng.uniform(5.0, 30.0)))),
         "trials": trials}
    if kind == "patch":
        c["n_rand"] = log(30_000, 300_000)
    if kind == "loop":
        c.update(precision="fp64" if rng.random() < 0.25 else "fp32", weighting="SNR" if rng.random() < 0.25 else "P-square",
                 row_variant=rng.random() < 0.7)
        if c["precision"] == "fp64":
            c["n_ps"] = min(c["n_ps"], 6_000_000 // n_ifg)
            c["cells"] = min(c["cells"], 96)
    return c


# ---------------------------------------------------------------- inputs ----
def _rng(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1_000_003 + salt * 7_919 + 17) % (1 << 62))


def _baselines(case, g):
    """Perpendicular baselines (f32 values) and the incidence that gives the trial count."""
    m, b = case["n_ifg"], 400.0 if case.get("n_ps", 0) > 1_000_000 else 300.0
    bp = (torch.rand(m, generator=g, device=DEV, dtype=torch.float64) * 2.0 - 1.0) * b
    bp = bp.float().double()
    span = float(bp.max() - bp.min())
    wraps = ((case["trials"] - 1) // 2 - 0.5) / 8.0
    topo = 20.0
    sin_inc = 2.0 * span * topo / (LAMBDA * RHO * wraps)
    if not 0.05 < sin_inc < 0.95:  # few interferograms or few trials: another height error
        sin_inc = 0.4
        topo = sin_inc * LAMBDA * RHO * wraps / (2.0 * span)
    return bp, math.asin(sin_inc), topo, wraps


def _scene(case, seed, salt=0):
    """A seeded patch on the device: deformation fields of 500 m correlation, DEM
    errors, 30 % stable candidates, the others random phase, a few pixels missing."""
    g = _rng(seed, salt)
    n, m, cells = case["n_ps"], case["n_ifg"], case["cells"]
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    side = CELL * cells + CELL / 2
    x, y = rand(n) * side, rand(n) * side
    # the corners keep the grid at cells x cells
    x[0], y[0], x[1], y[1] = 0.0, 0.0, side, side
    bp, inc, topo, wraps = _baselines(case, g)
    k_ps = ((rand(n) * 30.0 - 15.0) * (topo / 20.0) * 4.0 * math.pi / (LAMBDA * RHO * math.sin(inc))).float()
    grad = 1.0 + 0.02 * (x - x.mean()) / side
    if not case.get("row_variant", True):
        grad = torch.ones_like(grad)
    r = 256
    f = torch.fft.fftfreq(r, d=side / r, device=DEV)
    spec = torch.exp(-((f[:, None] ** 2 + f[None, :] ** 2) * (math.pi * 500.0) ** 2) / 2.0)
    fields = torch.empty(r * r, m, device=DEV)
    for c in range(m):
        v = torch.fft.ifft2(torch.fft.fft2(torch.randn(r, r, generator=g, device=DEV)) * spec).real
        fields[:, c] = (v / v.std() * (0.02 * 4.0 * math.pi / LAMBDA)).reshape(-1)
    at = (x / side * (r - 1)).round().long() * r + (y / side * (r - 1)).round().long()
    stable = rand(n) < 0.3
    ph = torch.empty(n, m, device=DEV, dtype=torch.complex64)
    bmat = torch.empty(n, m, device=DEV)
    for s in range(0, n, 250_000):
        e = min(n, s + 250_000)
        bmat[s:e] = (grad[s:e, None] * bp[None, :]).float()
        a = fields[at[s:e]] + k_ps[s:e, None] * bmat[s:e]
        noise = torch.where(stable[s:e, None], 0.3 * torch.randn(e - s, m, generator=g, device=DEV),
                            (torch.rand(e - s, m, generator=g, device=DEV) * 2.0 - 1.0) * math.pi)
        ph[s:e] = torch.polar(torch.ones_like(a), a + noise)
    missing = (rand(max(1, n // 10_000)) * n).long()
    ph[missing, (rand(missing.numel()) * m).long()] = 0.0
    d_a = rand(n) * 0.4 + 0.2
    ij = []
    for v in (y.float(), x.float()):
        b = torch.clamp(torch.ceil(((v - v.min()) + 1.0e-6) / CELL), min=1.0)
        ij.append(torch.where(b == b.max(), b - 1.0, b) if float(b.max()) > 1 else b)
    ij = torch.stack(ij, 1)
    n_i, n_j = int(ij[:, 0].max()), int(ij[:, 1].max())
    lin = (ij[:, 0].long() - 1) * n_j + (ij[:, 1].long() - 1)
    return {"ph": ph, "bperp": bmat, "bp": bp, "wraps": wraps, "inc": inc, "topo": topo, "x": x, "y": y, "D_A": d_a,
            "w0": 1.0 / d_a, "ij": ij, "lin": lin, "n_i": n_i, "n_j": n_j}


def _parms(case, topo=20.0):
    return {"filter_grid_size": CELL, "clap_win": 32.0, "clap_low_pass_wavelength": 800.0, "clap_alpha": 1.0, "clap_beta": 0.3,
            "max_topo_err": topo, "lambda": LAMBDA, "small_baseline_flag": "n",
            "filter_weighting": case.get("weighting", "P-square"), "gamma_change_convergence": 0.005,
            "gamma_max_iterations": 25}


def _low_pass():
    f = (np.arange(32) - 16.0) / (CELL * 32) * 800.0
    b = np.roll(1.0 / (1.0 + f ** 10), -16)
    return np.outer(b, b)


def _patch_dict(case, seed):
    """What the MAT files of a patch hold, in host memory (master image first)."""
    s = _scene(case, seed)
    n = case["n_ps"]
    ph = np.ones((n, case["n_ifg"] + 1), dtype=np.complex64)
    ph[:, 1:] = s["ph"].cpu().numpy()
    xy = np.stack([np.arange(1, n + 1), s["x"].cpu().numpy(), s["y"].cpu().numpy()], 1).astype(np.float32)
    return {"ph": ph, "bperp": np.concatenate([[0.0], s["bp"].cpu().numpy()]), "master_ix": 1,
            "bperp_mat": s["bperp"].double().cpu().numpy(), "D_A": s["D_A"].cpu().numpy(), "xy": xy,
            "mean_incidence": s["inc"], "parms": _parms(case, s["topo"]), "n_rand": case["n_rand"]}


def _histogram(bp, wraps, n_rand=20_000):
    return stage2.random_coherence_histogram(bp.cpu().numpy(), wraps, n_rand)


def _prepared(case, s, host=False):
    """The prepared patch and, for an upload from the device, its arrays there."""
    nr, top = _histogram(s["bp"], s["wraps"])
    none = np.zeros((0,), np.float32)
    inv = not case.get("row_variant", True)
    bperp = s["bperp"][0].contiguous() if inv else s["bperp"]
    amp = s["ph"].abs() + (s["ph"] == 0) if case.get("weighting") == "SNR" else s["x"].float()
    dev = {"ph_nm": s["ph"], "amp": amp, "bperp": bperp, "grid_lin": s["lin"].contiguous(),
           "weight0": s["w0"].contiguous(), "low_pass": torch.from_numpy(_low_pass()).to(DEV),
           "nr": torch.from_numpy(nr).to(DEV)}
    at = (lambda k: dev[k].cpu().numpy()) if host else (lambda k: none)  # noqa: E731
    p = stage2.PreparedPatch(
        n_ps=case["n_ps"], n_ifg=case["n_ifg"], ph_nm=at("ph_nm"), amp=at("amp"), bperp=at("bperp"), row_invariant=inv,
        bperp_nm=s["bp"].cpu().numpy(), grid_ij=s["ij"].cpu().numpy(), grid_lin=s["lin"].cpu().numpy(), n_i=s["n_i"],
        n_j=s["n_j"], weight0=s["w0"].cpu().numpy(), low_pass=_low_pass(), n_trial_wraps=s["wraps"], nr=nr, nr_max_nz_ix=top,
        low_coh_thresh=31, psquare=case.get("weighting", "P-square") == "P-square", gamma_change_convergence=0.005,
        gamma_max_iterations=25, clap_window=24, clap_alpha=1.0, clap_beta=0.3, grid_size=CELL)
    return p, dev


def _loaded(case, s, precision="fp32"):
    p, dev = _prepared(case, s)
    ctx = stage2.Stage2Context(0)
    torch.cuda.synchronize()  # the arrays are ready before the library's stream reads them
    ctx.load(p, precision, dev)
    return ctx


def _batch_cases(case):
    """The shapes of a batch: PS counts over their logarithm, 30 to 120 interferograms."""
    r = np.random.default_rng(2005 + case["patches"] * 31 + case["ps_lo"])
    out = []
    for k in range(case["patches"]):
        n = int(round(math.exp(r.uniform(math.log(case["ps_lo"]), math.log(case["ps_hi"])))))
        out.append({"n_ps": n, "n_ifg": int(r.integers(30, 121)), "cells": max(24, math.ceil(math.sqrt(n / 10.0))),
                    "trials": case["trials"]})
    return out


def _rows(case, seed):
    """Registry rows: a third of them coherent, and (topofit) one pixel in 500 missing."""
    g = _rng(seed)
    n, m = case["n_ps"], case["n_ifg"]
    bp, inc, topo, wraps = _baselines(case, g)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    noise = (rand(n, m) * 2.0 - 1.0) * math.pi
    if case["kind"] == "coherence":
        return torch.polar(torch.ones_like(noise), noise), bp, wraps
    bmat = bp[None, :] * (1.0 + 0.02 * (rand(n, 1) - 0.5))
    k = (rand(n, 1) - 0.5) * 2.0 * math.pi * wraps / float(bp.max() - bp.min())
    good = rand(n, 1) < 0.33
    noise = torch.where(good, 0.3 * torch.randn(n, m, generator=g, device=DEV, dtype=torch.float64), noise)
    z = torch.polar(torch.ones_like(noise), k * bmat + noise)
    z = torch.where(rand(n, m) < 0.002, torch.zeros_like(z), z)
    if case.get("single"):
        z, bmat = z.to(torch.complex64), bmat.float()
    return z, bmat, wraps


def prepare(case, seed):
    kind = case["kind"]
    if kind == "patch":
        return {"kind": kind, "patch": _patch_dict(case, seed)}
    if kind == "loop":
        return {"kind": kind, "ctx": _loaded(case, _scene(case, seed), case["precision"])}
    if kind == "batch":
        patches = [_prepared(c, _scene(c, seed, k + 1), host=True)[0] for k, c in enumerate(_batch_cases(case))]
        return {"kind": kind, "batch": batch.Batch(patches)}
    if kind == "gradient":
        s = _scene(case, seed)
        cmap = autograd.CoherenceMap(_prepared(case, s, host=True)[0])
        g = _rng(seed, 3)
        k = (torch.randn(case["n_ps"], generator=g, device=DEV) * 0.01).requires_grad_(True)
        gout = torch.rand(case["n_ps"], generator=g, device=DEV)
        return {"kind": kind, "map": cmap, "ph": s["ph"].requires_grad_(True), "K": k, "w": s["w0"].float(),
                "ab": [torch.tensor(v, dtype=torch.float64, device=DEV, requires_grad=True) for v in (1.1, 0.3)], "gout": gout}
    if kind == "stage3":
        s = _scene(case, seed)
        ctx = _loaded(case, s)
        ctx.run()
        coh = ctx.download(("coh_ps",))["coh_ps"]
        sel = np.flatnonzero(coh > np.quantile(coh, 0.7))
        # the selection leaves one interferogram in twelve out of the fit
        fit = np.array([c for c in range(case["n_ifg"]) if c % 12 != 5 or case["n_ifg"] < 12])
        return {"kind": kind, "ctx": ctx, "sel": sel, "fit": fit}
    if kind == "histogram":
        bp, _, _, wraps = _baselines(case, _rng(seed))
        return {"kind": kind, "bp": bp.cpu().numpy(), "wraps": wraps, "n_rand": case["n_rand"]}
    z, bp, wraps = _rows(case, seed)
    return {"kind": kind, "z": z.cpu().numpy(), "bp": bp.cpu().numpy(), "wraps": wraps}


def run(state):
    kind = state["kind"]
    if kind == "patch":
        r = stage2.run_stage2(state["patch"])
        return {k: r[k] for k in PM1 + ("i_loop", "gamma_change_save")}
    if kind == "loop":
        ctx = state["ctx"]
        ctx.reset()
        ctx.run()
        r = ctx.download(SUMMARY)
        return {k: r[k] for k in SUMMARY + ("i_loop", "gamma_change_save")}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        b.run()
        return [{k: r[k] for k in ("K_ps", "C_ps", "coh_ps", "N_opt", "i_loop")} for r in b.download()]
    if kind == "gradient":
        leaves = [state["ph"], state["K"], *state["ab"]]
        coh = autograd.coherence(state["map"], leaves[0], leaves[1], leaves[2], leaves[3], state["w"])
        return [coh.detach(), *torch.autograd.grad(coh, leaves, state["gout"])]
    if kind == "stage3":
        return stage3.reestimate_resident(state["ctx"], state["sel"], state["fit"], on_device=True)
    if kind == "histogram":
        nr, top = stage2.random_coherence_histogram(state["bp"], state["wraps"], state["n_rand"])
        return {"nr": nr, "top": top}
    if kind == "topofit":
        return list(kernels.run_stage2_topofit_kernel(state["z"], state["bp"], state["wraps"]))
    return kernels.run_stage2_topofit_coh_row_invariant_kernel(state["z"], state["bp"], state["wraps"])


# ------------------------------------------------------------------ work ----
def _sweep_flops(n, m, trials):
    return float(n) * m * (8 * trials + 32)  # the trial sums' complex multiply-adds and the refinement


def _clap_flops(cells, m):
    w = max(0, math.ceil(cells / 6) - 3) ** 2
    return w * m * 1.4e5


def work(case):
    kind = case["kind"]
    t = case["trials"]
    if kind == "batch":
        c = [_loop_work(x, 1) for x in _batch_cases(case)]
        return {"bytes": sum(x["bytes"] for x in c), "flops": sum(x["flops"] for x in c)}
    if kind == "histogram":
        return {"bytes": 8.0 * case["n_ifg"] + 808.0, "flops": _sweep_flops(case["n_rand"], case["n_ifg"], t)}
    n, m = case["n_ps"], case["n_ifg"]
    if kind in ("topofit", "coherence"):
        wide = 8 if kind == "topofit" and case["single"] else 16
        rows = n * m * (wide + (wide // 2 + 8 if kind == "topofit" else 0))
        return {"bytes": float(rows + n * 24), "flops": _sweep_flops(n, m, t)}
    if kind == "gradient":
        grid = float(case["cells"]) ** 2 * m
        return {"bytes": n * m * (8.0 + 4.0 + 8.0) + 24.0 * n, "flops": n * m * 150.0 + 4.0 * _clap_flops(case["cells"], m) + grid}
    if kind == "stage3":
        sel = 0.3 * n
        return {"bytes": sel * m * (8.0 + 4.0 + 8.0 + 4.0) + 8.0 * case["cells"] ** 2 * m,
                "flops": _sweep_flops(sel, m, t) + min(sel, case["cells"] ** 2) * m * 1.2e5}
    if kind == "patch":
        w = _loop_work(case, 5)
        return {"bytes": w["bytes"] + n * m * (8.0 + 8.0 + 4.0 + 8.0) + 8.0 * case["cells"] ** 2 * m,
                "flops": w["flops"] + _sweep_flops(case["n_rand"], m, t)}
    return _loop_work(case, 1)


def _loop_work(case, least):
    """At least `least` iterations over the rows, each read once an iteration."""
    n, m = case["n_ps"], case["n_ifg"]
    least = max(least, 3)  # the loop takes three iterations or more to meet its rule
    row = 8.0 + (4.0 if case.get("row_variant", True) else 0.0) + (4.0 if case.get("weighting") == "SNR" else 0.0)
    return {"bytes": least * n * m * row + 40.0 * n,
            "flops": least * (_sweep_flops(n, m, case["trials"]) + _clap_flops(case["cells"], m))}


# ----------------------------------------------------------------- exact ----
def _window_weight():
    r = np.arange(12.0)
    q = np.concatenate([r, r[::-1]])
    return (q[:, None] + q[None, :] + 1.0e-6) / 1024.0


def _clap(grid, n_i, n_j, alpha, beta):
    """CLAP of a [n_i * n_j, M] complex128 grid: 24-cell windows every 6 cells in 32 x 32
    transforms, gain max((smoothed |H| / median)^alpha - 1, 0) * beta + low pass, pyramid overlap-add."""
    m = grid.shape[1]
    nwi, nwj = math.ceil(n_i / 6) - 3, math.ceil(n_j / 6) - 3
    out = torch.zeros_like(grid)
    if nwi <= 0 or nwj <= 0:
        return out
    g7 = torch.from_numpy(np.exp(-0.5 * ((np.arange(7) - 3) / 1.2) ** 2)).to(DEV)
    low = torch.from_numpy(_low_pass()).to(DEV)
    pyramid = _window_weight()
    step = max(1, 40_000 // m)
    places = [(a, b) for a in range(nwi) for b in range(nwj)]
    total = torch.zeros_like(grid)
    for s in range(0, len(places), step):
        cells, weights = [], []
        for a, b in places[s:s + step]:
            r, c = max(0, 6 * a + 24 - n_i), max(0, 6 * b + 24 - n_j)
            i, j = np.arange(24) + 6 * a - r, np.arange(24) + 6 * b - c
            cells.append(i[:, None] * n_j + j[None, :])
            w = np.zeros((24, 24))
            w[r:, c:] = pyramid[:24 - r, :24 - c]
            weights.append(w)
        cells = torch.from_numpy(np.stack(cells)).to(DEV)
        weights = torch.from_numpy(np.stack(weights)).to(DEV)
        k = cells.shape[0]
        x = grid[cells.reshape(-1)].reshape(k, 24, 24, m).permute(0, 3, 1, 2)
        x = torch.fft.fft2(x, s=(32, 32))
        h = torch.fft.fftshift(x.abs(), dim=(-2, -1)).reshape(-1, 1, 32, 32)
        h = torch.nn.functional.conv2d(h, (g7[:, None] * g7[None, :])[None, None], padding=3).reshape(x.shape)
        h = torch.fft.ifftshift(h, dim=(-2, -1))
        srt = h.reshape(k, m, 1024).sort(dim=-1).values
        med = 0.5 * (srt[..., 511] + srt[..., 512])
        gain = torch.relu((h / torch.where(med != 0, med, 1.0)[..., None, None]) ** alpha - 1.0) * beta + low
        y = torch.fft.ifft2(x * gain)[..., :24, :24] * 1024.0 * weights[:, None]
        total = total.index_add(0, cells.reshape(-1), y.permute(0, 2, 3, 1).reshape(-1, m))
    return total


def _unit(f):
    a = f.abs()
    return torch.where(a > 0, f / torch.where(a > 0, a, 1.0), f)


def _sums(z, theta, half):
    """|sum_c z_c e^{-j theta_c t}| for t = -half .. half, [rows, trials]."""
    step = torch.polar(torch.ones_like(theta), -theta)
    w = z * torch.polar(torch.ones_like(theta), theta * half)
    out = torch.empty(z.shape[0], 2 * half + 1, dtype=torch.float64, device=DEV)
    for t in range(2 * half + 1):
        out[:, t] = w.sum(1).abs()
        w = w * step
    return out


def _refine(z, bp, mag, k0):
    """One weighted least-squares step from k0: K, C, coherence and the rotated row."""
    r = z * torch.polar(torch.ones_like(bp), -k0[:, None] * bp)
    ang = (r * r.sum(1).conj()[:, None]).angle()
    den = ((mag * bp) ** 2).sum(1)
    k = k0 + (mag * bp * mag * ang).sum(1) / torch.where(den != 0, den, 1.0)
    r = z * torch.polar(torch.ones_like(bp), -k[:, None] * bp)
    s, d = r.sum(1), mag.sum(1)
    return k, s.angle(), s.abs() / torch.where(d != 0, d, 1.0), r


def _span(bp, valid):
    lo = torch.where(valid, bp, math.inf).amin(1)
    hi = torch.where(valid, bp, -math.inf).amax(1)
    s = hi - lo
    return torch.where(torch.isfinite(s) & (s != 0), s, 1.0)


def _fit(z, bp, half):
    """The gamma loop's fit: first best trial, refined."""
    span = _span(bp, torch.ones_like(bp, dtype=torch.bool))
    best = _sums(z, bp / span[:, None] * (math.pi / 4), half).argmax(1)
    return _refine(z, bp, z.abs(), (math.pi / 4) / span * (best - half))


def _near_max(z, bp, half, tol=NEAR_MAX):
    """The registry's fit: every local maximum within tol of the best trial refined, the best of
    them kept (two candidates at the two ends: the better trial)."""
    valid = z != 0
    span, mag = _span(bp, valid), z.abs()
    den = mag.sum(1)
    v = _sums(z, bp / span[:, None] * (math.pi / 4), half) / torch.where(den != 0, den, 1.0)[:, None]
    pad = torch.full((v.shape[0], 1), -1.0, dtype=v.dtype, device=DEV)
    near = (v >= torch.cat([pad, v[:, :-1]], 1)) & (v >= torch.cat([v[:, 1:], pad], 1)) & (v >= v.amax(1, True) - tol)
    count, q = near.sum(1), (math.pi / 4) / span
    best = _refine(z, bp, mag, q * (v.argmax(1) - half))
    ends = (count == 2) & near[:, 0] & near[:, -1]
    left = near.clone()
    done = torch.zeros(v.shape[0], dtype=torch.bool, device=DEV)
    several = (count > 1) & ~ends
    for _ in range(int(count.max())):
        t = left.int().argmax(1)
        live = several & left.any(1)
        if not bool(live.any()):
            break
        f = _refine(z, bp, mag, q * (t - half))
        take = live & (~done | (f[2] > best[2]))
        best = tuple(torch.where(take if a.dim() == 1 else take[:, None], a, b) for a, b in zip(f, best))
        done |= take
        left[torch.arange(v.shape[0], device=DEV), t] = False
    return best


def _interp_taps():
    """The 79-tap interpolation filter of the P-square weighting (data of the method)."""
    text = (Path(stage2.__file__).parent / "csrc" / "interp10_taps.h").read_text()
    return np.array([float(v) for v in re.findall(r"[-+]?\d+\.\d+e[-+]\d+", text[text.index("{"):])])


def _psquare(coh, nr, top):
    """The weight of every row from the coherences' histogram against the random rows' (and Nr rescaled)."""
    d = (0.995 - 0.005) / 99.0
    b = torch.clamp(torch.ceil((coh - (0.005 + 0.015) / 2.0) / d), 0, 99).long()
    na = torch.bincount(b[torch.isfinite(coh)], minlength=100).double().cpu().numpy()
    nr = nr * (na[:31].sum() / nr[:31].sum())
    p = np.minimum(nr / np.where(na == 0, 1.0, na), 1.0)
    p[:31] = 1.0
    p[int(top):] = 0.0
    g = np.exp(-0.5 * ((np.arange(7) - 3) / 1.2) ** 2)
    smooth = np.convolve(np.concatenate([np.ones(7), p]), g)[7:107] / g.sum()
    wide = np.zeros(101 * 10)
    wide[::10] = np.concatenate([[1.0], smooth])
    lut = np.convolve(wide, _interp_taps() * 10.0)[39:39 + 1001]
    ix = torch.clamp(torch.floor(coh * 1000.0 + 0.5), 0, 1000).long()
    return (1.0 - torch.from_numpy(lut).to(DEV)[ix]) ** 2, nr


def _loop(s, case, nr, top, psquare):
    """The gamma loop to convergence in 64 bits."""
    n, m = s["ph"].shape
    half = (case["trials"] - 1) // 2
    K = torch.zeros(n, dtype=torch.float64, device=DEV)
    w, coh, was = s["w0"].clone(), torch.zeros(n, dtype=torch.float64, device=DEV), 0.0
    order = torch.argsort(s["lin"])
    step = max(1_000, 24_000_000 // m)
    res = {}
    for loop in range(1, 26):
        grid = torch.zeros(s["n_i"] * s["n_j"], m, dtype=torch.complex128, device=DEV)
        for a in range(0, n, step):
            at = order[a:a + step]
            kk = torch.where(torch.isnan(K[at]), torch.nan, K[at])
            ramp = torch.polar(torch.ones(at.numel(), m, dtype=torch.float64, device=DEV), -kk[:, None] * s["bperp"][at].double())
            grid.index_add_(0, s["lin"][at], s["ph"][at].to(torch.complex128) * ramp * w[at, None])
        clean = torch.where(torch.isnan(grid.real) | torch.isnan(grid.imag), 0.0, grid)
        filt = _unit(_clap(clean, s["n_i"], s["n_j"], 1.0, 0.3))
        K2, C2, coh2 = torch.empty_like(K), torch.empty_like(K), torch.empty_like(K)
        keep = {"K": K, "w": w, "grid": grid, "filt": filt}
        bad = torch.empty(n, dtype=torch.bool, device=DEV)
        for a in range(0, n, step):
            z = filt[s["lin"][a:a + step]].conj() * s["ph"][a:a + step].to(torch.complex128)
            K2[a:a + step], C2[a:a + step], coh2[a:a + step], r = _fit(z, s["bperp"][a:a + step].double(), half)
            bad[a:a + step] = (z == 0).any(1)
            if not psquare:
                ang = r.angle()
                ang[bad[a:a + step]] = 0.0
                amp = s["ph"][a:a + step].abs().double()
                amp = torch.where(amp == 0, 1.0, amp)
                g, a2 = (amp * ang.cos()).mean(1), (amp * amp).mean(1)
                sig = torch.sqrt(0.5 * (a2 - g * g))
                res.setdefault("w", torch.empty_like(w))[a:a + step] = torch.where(sig != 0, g / torch.where(sig != 0, sig, 1.0), 0.0)
        K2[bad], C2[bad], coh2[bad] = math.nan, 0.0, 0.0
        rms = float(((coh2 - coh) ** 2).mean().sqrt())
        delta, was = rms - was, rms
        K, coh = K2, coh2
        if abs(delta) < 0.005:
            break
        if psquare:
            w, nr = _psquare(coh, nr, top)
        else:
            w = res["w"].clone()
    return {"K_ps": K, "C_ps": C2, "coh_ps": coh, "coh_ps_save": coh, "N_opt": (~bad).double(), "Nr": nr, "i_loop": loop,
            "gamma_change_save": was, "used": keep}


def _to_host(d, names):
    return {k: (d[k].cpu().numpy() if torch.is_tensor(d[k]) else d[k]) for k in names}


def exact(case, seed):
    kind = case["kind"]
    if kind == "histogram":
        return None  # whole numbers of one serial random stream
    if kind == "loop":
        s = _scene(case, seed)
        nr, top = _histogram(s["bp"], s["wraps"])
        return _to_host(_loop(s, case, nr, top, case["weighting"] == "P-square"), SUMMARY + ("i_loop", "gamma_change_save"))
    if kind == "patch":
        s = _scene(case, seed)
        nr, top = _histogram(s["bp"], s["wraps"], case["n_rand"])
        r = _loop(s, case, nr, top, True)
        u, m = r.pop("used"), case["n_ifg"]
        z = u["filt"][s["lin"]].conj() * s["ph"].to(torch.complex128)
        bp = s["bperp"].double()
        ang = (z * torch.polar(torch.ones_like(bp), -torch.nan_to_num(r["K_ps"])[:, None] * bp)).angle()
        ang[r["N_opt"] == 0] = 0.0
        r["ph_res"], r["ph_patch"] = ang, u["filt"][s["lin"]]
        r["ph_weight"] = s["ph"].to(torch.complex128) * torch.polar(torch.ones_like(bp), -u["K"][:, None] * bp) * u["w"][:, None]
        r["ph_grid"] = u["grid"].reshape(s["n_i"], s["n_j"], m)
        return _to_host(r, PM1 + ("i_loop", "gamma_change_save"))
    if kind == "batch":
        out = []
        for k, c in enumerate(_batch_cases(case)):
            s = _scene(c, seed, k + 1)
            out.append(_to_host(_loop(s, c, *_histogram(s["bp"], s["wraps"]), True), ("K_ps", "C_ps", "coh_ps", "N_opt", "i_loop")))
        return out
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "stage3":
        return _exact_stage3(case, seed)
    z, bp, wraps = _rows(case, seed)
    half = math.ceil(8.0 * wraps)
    z, bp = z.to(torch.complex128), bp.double()
    bp = bp if bp.dim() == 2 else bp[None, :].expand(z.shape[0], -1)
    k, c, coh, r = _near_max(z, bp, half)
    if kind == "coherence":
        return coh.cpu().numpy()
    return [v.cpu().numpy() for v in (k, c, coh, r)]


def _exact_gradient(case, seed):
    st = prepare(case, seed)
    s = _scene(case, seed)
    ph = st["ph"].detach().to(torch.complex128).requires_grad_(True)
    k = st["K"].detach().double().requires_grad_(True)
    al, be = (v.detach().clone().requires_grad_(True) for v in st["ab"])
    bp = s["bperp"].double()
    e = torch.polar(torch.ones_like(bp), -k[:, None] * bp)
    grid = torch.zeros(s["n_i"] * s["n_j"], ph.shape[1], dtype=torch.complex128, device=DEV)
    grid = grid.index_add(0, s["lin"], ph * e * st["w"].double()[:, None])
    f = _clap(grid, s["n_i"], s["n_j"], al, be)[s["lin"]]
    a = f.abs()
    z = torch.where(a > 0, f / torch.where(a > 0, a, 1.0), 0.0).conj() * ph
    d = z.abs().sum(1)
    coh = (z * e).sum(1).abs() / torch.where(d > 0, d, 1.0)
    return [coh.detach(), *torch.autograd.grad(coh, [ph, k, al, be], st["gout"].double())]


def _exact_stage3(case, seed):
    st = prepare(case, seed)
    s = _scene(case, seed)
    n_i, n_j, m = s["n_i"], s["n_j"], case["n_ifg"]
    half = (case["trials"] - 1) // 2
    grid = torch.from_numpy(st["ctx"].download(("ph_grid",))["ph_grid"]).to(DEV).to(torch.complex128)
    grid = torch.where(torch.isnan(grid.real) | torch.isnan(grid.imag), 0.0, grid)
    sel = torch.from_numpy(st["sel"]).to(DEV)
    cells, job = torch.unique(s["lin"][sel], return_inverse=True)
    ci, cj = cells // n_j + 1, cells % n_j + 1
    i0, j0 = torch.clamp(ci - 16, min=1), torch.clamp(cj - 16, min=1)
    i0, j0 = torch.where(i0 + 31 > n_i, n_i - 31, i0), torch.where(j0 + 31 > n_j, n_j - 31, j0)
    fits = (i0 >= 1) & (j0 >= 1)
    g7 = torch.from_numpy(np.exp(-0.5 * ((np.arange(7) - 3) / 1.2) ** 2)).to(DEV)
    low = torch.from_numpy(_low_pass()).to(DEV)
    value = torch.zeros(cells.numel(), m, dtype=torch.complex128, device=DEV)
    step, r32 = max(1, 60_000 // m), torch.arange(32, device=DEV)
    for a in range(0, cells.numel() if bool(fits.any()) else 0, step):
        e = min(cells.numel(), a + step)
        ii, jj = i0[a:e, None] - 1 + r32, j0[a:e, None] - 1 + r32
        x = grid[ii.clamp(0, n_i - 1)[:, :, None], jj.clamp(0, n_j - 1)[:, None, :]]  # [cells, 32, 32, m]
        own, k = (ci - i0)[a:e], torch.arange(e - a, device=DEV)
        oj = (cj - j0)[a:e]
        x[k, own.clamp(0, 31), oj.clamp(0, 31)] = 0.0
        x = torch.fft.fft2(x.permute(0, 3, 1, 2))
        h = torch.fft.fftshift(x.abs(), dim=(-2, -1)).reshape(-1, 1, 32, 32)
        h = torch.nn.functional.conv2d(h, (g7[:, None] * g7[None, :])[None, None], padding=3).reshape(x.shape)
        h = torch.fft.ifftshift(h, dim=(-2, -1))
        srt = h.reshape(e - a, m, 1024).sort(dim=-1).values
        med = 0.5 * (srt[..., 511] + srt[..., 512])
        gain = torch.relu(h / torch.where(med != 0, med, 1.0)[..., None, None] - 1.0) * 0.3 + low
        value[a:e] = torch.fft.ifft2(x * gain)[k, :, own.clamp(0, 31), oj.clamp(0, 31)]
    value[~fits] = 0.0
    patch = value[job]
    psd = s["ph"][sel].to(torch.complex128) * patch.conj()
    bad = (psd == 0).any(1)
    fit = torch.from_numpy(st["fit"]).to(DEV)
    z, bp = _unit(psd)[:, fit], s["bperp"][sel][:, fit].double()
    parts = [_near_max(z[a:a + 200_000], bp[a:a + 200_000], half) for a in range(0, sel.numel(), 200_000)]
    k, c, coh, r = (torch.cat(v) for v in zip(*parts))
    k[bad], c[bad], coh[bad] = math.nan, 0.0, math.nan
    res = torch.zeros(sel.numel(), m, dtype=torch.float64, device=DEV)
    res[:, fit] = torch.where(bad[:, None], 0.0, r.angle())
    return {"ph_patch2": patch, "K_ps2": k, "C_ps2": c, "coh_ps2": coh, "ph_res2": res}
