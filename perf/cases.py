"""The work that users of this framework have it do, as cases that a timer can run.

Four kinds, each through the framework's public entry points:

  solve    the isolated Poisson solve on device buffers (SpectralSolver.solve), in its three
           precisions, with and without the potential map; bin sides are powers of two, square
           and not, as the library takes them (16 to 4096);
  run      a placement resumed from a checkpoint for a few iterations, then its positions
           (erp_restore, Placement.step, erp_get_positions);
  host     the drop-in form for a program that owns the coordinates: a loop of
           Placement.step_host over pinned arrays, statistics read after every step;
  batch    many designs advanced together (Batch): resumed, run, and every design's positions.

A `spread` of 0 is the jittered centre start of a fresh placement, where nearly all cells share a
few bins; otherwise the movable cells start uniformly spread over that share of the die's width,
as a placement does that keeps its design's coordinates, or one that is well under way.

The loop grows a difference of one rounding by a factor of a few in every iteration, so a pass is
a few iterations from a fixed state, not a whole placement: its outputs can then be compared.
"""
import ctypes as C
import math

import numpy as np
import torch

import reda_erplacer_gb300 as R
from reda_erplacer_gb300 import lib as L
from reda_erplacer_gb300.placement import Batch, Placement, SpectralSolver

PRECISION = {"fp32": L.PREC_FP32, "tf32": L.PREC_TF32_GEMM, "bf16x3": L.PREC_BF16X3_GEMM}


def listed():
    return [
        # the smallest solve: three short launches, as a small block's placer issues them
        {"name": "solve-64x64", "kind": "solve", "m": 64, "n": 64, "precision": "fp32", "psi": False},
        # the grid of the 1M-cell workload, fields only, as every iteration solves it
        {"name": "solve-1024", "kind": "solve", "m": 1024, "n": 1024, "precision": "fp32", "psi": False},
        # the largest grids the library takes, not square, with the potential (energy asked for)
        {"name": "solve-4096x2048-psi", "kind": "solve", "m": 4096, "n": 2048, "precision": "fp32", "psi": True},
        # the tensor-core forms: TF32 at an ordinary oblong grid, BF16x3 at a large one with the potential
        {"name": "solve-1024x512-tf32", "kind": "solve", "m": 1024, "n": 512, "precision": "tf32", "psi": False},
        {"name": "solve-2048-bf16x3-psi", "kind": "solve", "m": 2048, "n": 2048, "precision": "bf16x3", "psi": True},
        # a small block: every iteration is a chain of short kernels
        {"name": "run-2k", "kind": "run", "cells": 2003, "macros": 3, "m": 64, "n": 64, "precision": "fp32",
         "spread": 0.0, "steps": 8},
        # the 20,000-cell workload on its grid, from the jittered start
        {"name": "run-20k", "kind": "run", "cells": 20000, "macros": 0, "m": 256, "n": 256, "precision": "fp32",
         "spread": 0.0, "steps": 6},
        # a mid-sized design half spread, on an oblong grid
        {"name": "run-200k", "kind": "run", "cells": 200001, "macros": 9, "m": 512, "n": 1024, "precision": "fp32",
         "spread": 0.5, "steps": 4},
        # the 1M-cell workload with its cells spread over the die, where most of its iterations are
        {"name": "run-1m", "kind": "run", "cells": 1000000, "macros": 16, "m": 1024, "n": 1024, "precision": "fp32",
         "spread": 0.95, "steps": 3},
        # the tensor-core solve inside the loop, on the default 512 x 512 bins
        {"name": "run-60k-bf16x3", "kind": "run", "cells": 60000, "macros": 4, "m": 512, "n": 512,
         "precision": "bf16x3", "spread": 0.6, "steps": 4},
        # the drop-in loop: coordinates in pinned host memory, the default 512 x 512 bins
        {"name": "host-100k", "kind": "host", "cells": 100000, "macros": 5, "m": 512, "n": 512, "spread": 0.3, "steps": 4},
        # a batch of small and mid-sized designs, from the jittered start
        {"name": "batch-32", "kind": "batch", "count": 32, "least": 2000, "most": 60000, "spread": 0.0, "steps": 8},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "run", "run", "run", "host", "batch"))
    spread = rng.choice((0.0, round(rng.uniform(0.1, 0.95), 3)))
    if kind == "solve":
        precision = rng.choice(("fp32", "fp32", "tf32", "bf16x3"))
        low, high = (4, 12) if precision == "fp32" else (7, 11)   # the transform matrices of the others are dense
        m, n = 2 ** rng.randint(low, high), 2 ** rng.randint(low, high)
        if m * n > 4096 * 2048:
            m = m // 2
        # a bin's aspect ratio is a free number of the solve
        return {"kind": kind, "m": m, "n": n, "precision": precision, "psi": rng.random() < 0.4,
                "bin_w": round(rng.uniform(0.5, 2.0), 3)}
    if kind == "batch":
        least = int(_log(rng, 1000, 4000))
        return {"kind": kind, "count": rng.randint(2, 32), "least": least, "most": int(_log(rng, 2 * least, 60000)),
                "spread": spread, "steps": rng.randint(4, 8)}
    cells = int(_log(rng, 1500, 1000000 if kind == "run" else 100000))
    b = int(round(math.log2(math.sqrt(cells) / 2)))
    m, n = (2 ** min(max(b + rng.choice((0, 0, 1)), 6), 10) for _ in range(2))
    case = {"kind": kind, "cells": cells, "macros": rng.randint(0, 16), "m": m, "n": n, "spread": spread,
            "steps": rng.randint(3, 7) if m * n <= 256 * 256 else rng.randint(2, 4)}
    if kind == "run":
        case["precision"] = rng.choice(("fp32", "fp32", "bf16x3")) if min(m, n) >= 128 else "fp32"
    return case


# ---- inputs ----

def _density(m, n, seed):
    """A density map as the isolated-solve workload has it: a 0.7 background, Gaussian blobs of the cells,
    and macro blocks at 1.0; made on the GPU."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g = torch.Generator().manual_seed(int(seed) * 7919 + m * 31 + n)
    u = torch.rand(48, 5, generator=g, dtype=torch.float64)
    x = (torch.arange(m, dtype=torch.float64, device=dev) + 0.5) / m
    y = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n
    cx, cy, s, amp = (u[:, k, None].to(dev) for k in range(4))
    s = 0.005 + 0.06 * s
    gx = torch.exp(-((x[None, :] - cx) / s) ** 2 / 2) * (0.1 + 0.4 * amp)
    gy = torch.exp(-((y[None, :] - cy) / s) ** 2 / 2)
    rho = 0.7 + gx.T @ gy
    rho += 0.05 * torch.rand(m, n, generator=g, dtype=torch.float32).to(dev)
    for k in range(10):
        i, j = int(u[k, 0] * 0.9 * m), int(u[k, 1] * 0.9 * n)
        w, h = max(1, int((0.03 + 0.09 * u[k, 2]) * m)), max(1, int((0.03 + 0.09 * u[k, 4]) * n))
        rho[i:i + w, j:j + h] = 1.0
    return rho.float().contiguous()


def _design(cells, macros, spread, seed):
    """The synthetic netlist of a case, with its movable cells spread as the case says."""
    d = R.synth(cells, int(round(1.05 * cells)), num_io=max(4, cells // 250), num_macros=macros,
                macro_area_frac=0.015, utilization=0.65, seed=1000 + int(seed))
    if spread > 0:
        g, k = np.random.default_rng(int(seed) + 77), d.num_movable
        for c, s, die in ((d.x, d.w, d.die_w), (d.y, d.h, d.die_h)):
            at = die / 2 - s[:k] / 2 + spread * die * (g.random(k) - 0.5)
            c[:k] = np.clip(at, 0, die - s[:k] - 1).astype(np.float32)
    return d


def _members(case, seed):
    """(cells, macros, bins, seed) of each design of a batch case: sizes spread evenly over their logarithm."""
    out, ratio = [], case["most"] / case["least"]
    for i in range(case["count"]):
        cells = int(round(case["least"] * ratio ** ((i * 7 % case["count"] + 0.5) / case["count"])))
        out.append((cells, i * 5 % 17, R.bins_for_cells(cells), int(seed) * 100 + i))
    return out


def _pinned(count, dtype=np.float32):
    return torch.empty(count * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)


class _Saved:
    """A context's checkpoint in pinned host memory."""

    def __init__(self, ctx):
        self.ctx, n = ctx, C.c_size_t()
        L.check(L.load().erp_checkpoint_size(ctx, C.byref(n)), ctx)
        self.blob = _pinned(n.value, np.uint8)
        L.check(L.load().erp_checkpoint(ctx, self.blob.ctypes.data, n.value), ctx)

    def restore(self):
        L.check(L.load().erp_restore(self.ctx, self.blob.ctypes.data, self.blob.nbytes), self.ctx)


def _read_positions(ctx, x, y):
    L.check(L.load().erp_get_positions(ctx, x.ctypes.data_as(L.f32p), y.ctypes.data_as(L.f32p)), ctx)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        m, n = case["m"], case["n"]
        rho = _density(m, n, seed)
        out = [torch.empty_like(rho) for _ in range(3 if case["psi"] else 2)]
        solver = SpectralSolver(m, n, case.get("bin_w", 1.0), 1.0, stream=torch.cuda.current_stream().cuda_stream,
                                precision=PRECISION[case["precision"]])
        return {"kind": kind, "solver": solver, "rho": rho, "out": out}
    if kind == "batch":
        parts = _members(case, seed)
        designs = [_design(c, k, case["spread"], s) for c, k, _, s in parts]
        batch = Batch(designs, [(b, b) for _, _, b, _ in parts], 1.0, start_mode=L.START_DB)
        ctx = [C.c_void_p(batch.lib.erp_batch_context(batch.h, i)) for i in range(len(designs))]
        ends = np.cumsum([d.num_nodes for d in designs])
        x, y = _pinned(int(ends[-1])), _pinned(int(ends[-1]))
        return {"kind": kind, "batch": batch, "ctx": ctx, "saved": [_Saved(c) for c in ctx], "x": x, "y": y,
                "parts": list(zip(np.split(x, ends[:-1]), np.split(y, ends[:-1]))), "steps": case["steps"]}
    d = _design(case["cells"], case["macros"], case["spread"], seed)
    p = Placement(d, (case["m"], case["n"]), 1.0, start_mode=L.START_DB,
                  precision=PRECISION[case.get("precision", "fp32")])
    return {"kind": kind, "placement": p, "steps": case["steps"], "saved": _Saved(p.h), "start": (d.x, d.y),
            "x": _pinned(d.num_nodes), "y": _pinned(d.num_nodes)}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        state["solver"].solve(state["rho"].data_ptr(), *(t.data_ptr() for t in state["out"]))
        return state["out"]
    x, y = state["x"], state["y"]
    if kind == "batch":
        for s in state["saved"]:
            s.restore()
        done, last = state["batch"].run(state["steps"])
        for c, (u, v) in zip(state["ctx"], state["parts"]):
            _read_positions(c, u, v)
        return {"x": x, "y": y, "iterations": np.array(done), "stats": np.array([_stats(t) for t in last])}
    p = state["placement"]
    state["saved"].restore()
    if kind == "host":
        x[:], y[:] = state["start"]
        for _ in range(state["steps"]):
            last = p.step_host(x, y)
        return {"x": x, "y": y, "iterations": last["iteration"] + 1, "stats": _stats(last)}
    for _ in range(state["steps"] - 1):
        p.step(stats=False)
    p.step()
    _read_positions(p.h, x, y)
    return {"x": x, "y": y, "iterations": p.last_stats["iteration"] + 1, "stats": _stats(p.last_stats)}


def _stats(last):
    return np.array([last[k] for k in ("hpwl", "overflow", "density_weight", "gamma", "alpha")], np.float32)


# ---- the work of a pass ----

def _step_work(cells, macros, m, n):
    """Bytes and operations of one placement step: what each pass of the loop has to read and write once
    (indices and floats of 4 bytes, 64-bit sums of the density map, the transforms' intermediates)."""
    nets = int(round(1.05 * cells))
    pins = 4.81 * nets + max(4, cells // 250)   # the netlist's degree mix
    bins = float(m * n)
    wire = 28 * pins + 4 * nets + 12 * pins + 12 * cells
    density = 28 * cells + 8 * bins
    solve = 44 * bins
    force = 36 * cells + 8 * bins
    update = 76 * cells
    flops = 60 * pins + 60 * cells + 15 * bins * (math.log2(m) + math.log2(n))
    return wire + density + solve + force + update, flops


def work(case):
    kind = case["kind"]
    if kind == "solve":
        m, n, maps = case["m"], case["n"], 3 if case["psi"] else 2
        bins = float(m * n)
        if case["precision"] == "fp32":   # rho in, the spectra between the axes, the fields out
            return {"bytes": 4 * bins * (1 + maps), "flops": 2.5 * bins * (1 + maps) * (math.log2(m) + math.log2(n))}
        products = 1 if case["precision"] == "tf32" else 3
        return {"bytes": 4 * bins * (1 + maps), "flops": 2 * products * bins * (1 + maps) * (m + n)}
    if kind == "batch":   # the mean size of a log-uniform draw
        a, b = case["least"], case["most"]
        cells = (b - a) / math.log(b / a)
        side = R.bins_for_cells(cells)
        by, fl = _step_work(cells, 8, side, side)
        return {"bytes": by * case["count"] * case["steps"], "flops": fl * case["count"] * case["steps"]}
    by, fl = _step_work(case["cells"], case["macros"], case["m"], case["n"])
    by, fl = by * case["steps"], fl * case["steps"]
    if kind == "host":
        by += 16 * case["cells"] * case["steps"]
    return {"bytes": by, "flops": fl}


# ---- the same in 64 bits ----

def _axis(n, kind, dev):
    """The transform along one axis as a matrix: cosine analysis, or the cosine or sine synthesis."""
    i, u = torch.arange(n, dtype=torch.float64, device=dev), torch.arange(n, dtype=torch.float64, device=dev)
    # (2 i + 1) u modulo 4 n: the angle stays small, so its 64-bit sine is exact to the last bits
    a = torch.remainder((2 * i[:, None] + 1) * u[None, :], 4 * n) * (math.pi / (2 * n))
    if kind == "analysis":
        return torch.cos(a).T * (2.0 / n)
    c = torch.full((n,), 2.0, dtype=torch.float64, device=dev)
    c[0] = 1.0
    return (torch.cos(a) if kind == "cos" else torch.sin(a)) * c[None, :]


def _poisson(rho, bin_w, bin_h, psi):
    m, n = rho.shape
    dev = rho.device
    A = _axis(m, "analysis", dev) @ rho @ _axis(n, "analysis", dev).T
    wu = torch.arange(m, dtype=torch.float64, device=dev)[:, None] * (2 * math.pi / m)
    wv = torch.arange(n, dtype=torch.float64, device=dev)[None, :] * (2 * math.pi / n) * (bin_w / bin_h)
    k2 = wu * wu + wv * wv
    k2[0, 0] = 1.0
    A = A / k2
    A[0, 0] = 0.0
    cm, cn = _axis(m, "cos", dev), _axis(n, "cos", dev)
    out = [_axis(m, "sin", dev) @ (A * wu / 2) @ cn.T, cm @ (A * wv / 2) @ _axis(n, "sin", dev).T]
    return out + [cm @ A @ cn.T] if psi else out


def _wirelength(t, x, y, gamma):
    """Weighted-average wirelength gradient per cell and the total half-perimeter."""
    hpwl, grads = 0.0, []
    for v, off, die in ((x, t["pin_ox"], t["die_w"]), (y, t["pin_oy"], t["die_h"])):
        p = v[t["pin_inst"]] + off
        q, net, E = p[t["net_pins"]], t["pin_net"], t["E"]
        big = torch.zeros(E, dtype=torch.float64, device=v.device).scatter_reduce(0, net, q, "amax", include_self=False)
        low = torch.zeros(E, dtype=torch.float64, device=v.device).scatter_reduce(0, net, q, "amin", include_self=False)
        two = torch.arange(E, device=v.device) < t["n_2nets"]
        big = torch.where(two, big, big.clamp(min=0.0))
        low = torch.where(two, low, low.clamp(max=die + 1.0))
        hpwl = hpwl + (big - low).sum()
        g = 0.0
        for sign, e in ((1.0, torch.exp((q - big[net]) / gamma)), (-1.0, torch.exp((low[net] - q) / gamma))):
            s = torch.zeros(E, dtype=torch.float64, device=v.device).index_add_(0, net, e)
            w = torch.zeros(E, dtype=torch.float64, device=v.device).index_add_(0, net, e * q)
            b = sign / (gamma * s)
            a = (1 - b * w) / s
            g = g + sign * (a[net] + b[net] * q) * e
        per_pin = torch.zeros(len(p), dtype=torch.float64, device=v.device)
        per_pin[t["net_pins"]] = g
        grads.append(torch.zeros(len(v), dtype=torch.float64, device=v.device).index_add_(0, t["pin_inst"], per_pin))
    return grads[0][:t["k"]], grads[1][:t["k"]], hpwl


def _overlaps(at, size, step, bins, first, count):
    """For each cell the first `count` bins from `first`: their indices, and the signed overlaps."""
    k = first[:, None] + torch.arange(count, device=at.device)
    return k, torch.minimum(at[:, None] + size[:, None], (k + 1) * step) - torch.maximum(at[:, None], k * step)


def _place(case, d, steps):
    """`steps` iterations of the electrostatic placement loop in 64 bits."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
    i = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.int64)  # noqa: E731
    m, n, k = case["m"], case["n"], d.num_movable
    deg = np.diff(d.net_ptr)
    t = {"pin_ox": f(d.pin_ox), "pin_oy": f(d.pin_oy), "pin_inst": i(d.pin_inst), "net_pins": i(d.net_pins),
         "pin_net": i(np.repeat(np.arange(d.num_nets), deg)), "E": d.num_nets, "n_2nets": d.n_2nets, "k": k,
         "die_w": float(d.die_w), "die_h": float(d.die_h)}
    x, y, w, h, pins = f(d.x), f(d.y), f(d.w), f(d.h), f(d.num_pins_f)[:k]
    bw, bh = d.die_w / m, d.die_h / n
    # fixed cells: their exact overlap with every bin (the last row and column of bins stay empty)
    base = torch.zeros(m, n, dtype=torch.float64, device=dev)
    for c in range(k, d.num_nodes):
        if d.w[c] > 0 and d.h[c] > 0:
            both = []
            for at, size, step, bins in ((float(d.x[c]), float(d.w[c]), bw, m), (float(d.y[c]), float(d.h[c]), bh, n)):
                e = torch.arange(bins, dtype=torch.float64, device=dev) * step
                o = (torch.clamp(e + step, max=at + size) - torch.clamp(e, min=at)).clamp(min=0)
                o[-1] = 0.0
                both.append(o)
            base += both[0][:, None] * both[1][None, :]
    w, h = w[:k], h[:k]
    cw, ch = torch.clamp(w, min=bw * math.sqrt(2)), torch.clamp(h, min=bh * math.sqrt(2))
    ratio, ox, oy = w * h / (cw * ch), (w - cw) / 2, (h - ch) / 2
    nx, ny = int(math.ceil(float(cw.max()) / bw)) + 2, int(math.ceil(float(ch.max()) / bh)) + 2
    px, py = x[:k].clone(), y[:k].clone()
    pgx, pgy = torch.zeros_like(px), torch.zeros_like(py)
    base_gamma = gamma = 4.0 * (bw + bh)
    dw, alpha, cur, first = 8e-5, 1.0, 0.0, None
    for it in range(steps):
        wx, wy, hpwl = _wirelength(t, x, y, gamma)
        hpwl = float(hpwl)
        ax, ay = x[:k] + ox, y[:k] + oy
        ix, vx = _overlaps(ax, cw, bw, m, torch.floor(ax / bw).clamp(-1, m).long().clamp(min=0), nx)
        iy, vy = _overlaps(ay, ch, bh, n, torch.floor(ay / bh).clamp(-1, n).long().clamp(min=0), ny)
        rho = torch.zeros(m * n, dtype=torch.float64, device=dev)
        for a in range(nx):
            for b in range(ny):
                v = ratio * vx[:, a].clamp(min=0) * vy[:, b].clamp(min=0)
                ok = (ix[:, a] < m - 1) & (iy[:, b] < n - 1)
                rho.index_add_(0, torch.where(ok, ix[:, a] * n + iy[:, b], 0), torch.where(ok, v, 0.0))
        rho = rho.view(m, n) + base
        overflow = float((rho - bw * bh).clamp(min=0).sum()) / float(np.float32(d.movable_area))
        fx, fy = _poisson(rho / (bw * bh), bw, bh, False)
        # the force: bins from the truncated lower edge to the truncated upper edge, overlaps not clamped
        ux, uy = torch.trunc((ax + cw) / bw).long() + 1, torch.trunc((ay + ch) / bh).long() + 1
        gx, gy = torch.zeros_like(px), torch.zeros_like(py)
        for a in range(nx):
            for b in range(ny):
                ok = (ix[:, a] < ux.clamp(max=m)) & (iy[:, b] < uy.clamp(max=n))
                at = torch.where(ok, ix[:, a] * n + iy[:, b], 0)
                area = torch.where(ok, vx[:, a] * vy[:, b], 0.0)
                gx += area * fx.reshape(-1)[at]
                gy += area * fy.reshape(-1)[at]
        gx, gy = -gx * ratio, -gy * ratio
        last_alpha = alpha
        alpha = (1 + math.sqrt(4 * alpha * alpha + 1)) / 2
        beta = (last_alpha - 1) / alpha
        if it == 0:
            dw *= float(wx.abs().sum() + wy.abs().sum()) / float(gx.abs().sum() + gy.abs().sum())
        pre = 1 / torch.clamp(pins + dw * w * h, max=1.0)
        gx, gy = (wx + dw * gx) * pre, (wy + dw * gy) * pre
        if it > 0:
            alpha = math.sqrt(float(((x[:k] - px) ** 2 + (y[:k] - py) ** 2).sum())
                              / float(((gx - pgx) ** 2 + (gy - pgy) ** 2).sum()))
        for v, p, g, size, die in ((x, px, gx, w, t["die_w"]), (y, py, gy, h, t["die_h"])):
            new = v[:k] + beta * (v[:k] - p) - alpha * g
            p.copy_(v[:k])
            v[:k] = torch.minimum(new.clamp(min=0), die - size - 1)
        pgx, pgy = gx, gy
        stats = [hpwl, overflow, dw, gamma, alpha]
        first = hpwl if first is None else first
        delta, cur = hpwl - cur, hpwl
        power = max(0.9999 ** (it + 1), 0.98) if delta < 0 else min(max(1.05 ** (-delta / first), 0.95), 1.05)
        dw *= 1.05 * power
        gamma = base_gamma * min(max(10.0 ** ((overflow - 0.1) * 20 / 9 - 1), 0.05), 10.0)
    return {"x": x.cpu(), "y": y.cpu(), "iterations": None, "stats": torch.tensor(stats, dtype=torch.float64)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return _poisson(_density(case["m"], case["n"], seed).double(), case.get("bin_w", 1.0), 1.0, case["psi"])
    if kind == "batch":
        every = [_place(dict(m=b, n=b), _design(c, k, case["spread"], s), case["steps"])
                 for c, k, b, s in _members(case, seed)]
        return {"x": torch.cat([e["x"] for e in every]), "y": torch.cat([e["y"] for e in every]), "iterations": None,
                "stats": torch.stack([e["stats"] for e in every])}
    return _place(case, _design(case["cells"], case["macros"], case["spread"], seed), case["steps"])
