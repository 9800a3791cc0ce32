"""The calls that programs using regridding_gb300 spend their time in, as
cases that can be timed and compared: each is one pass through public entry
points, on inputs made from a seed.

Grids are the package's synthetic family (``workloads.grid_pair``): a
vertex grid on [-1, 1]^2, rotated and sinusoidally distorted, against a
rectilinear grid over roughly the same square whose vertices carry a small
jitter.  ``exact`` restates every computed output in 64 bits with torch or
numpy alone.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import regridding_gb300 as rg
from regridding_gb300 import autograd, batching

F64 = torch.float64


def listed():
    return [
        # the first call of the README on a small detector cut-out: numpy in,
        # numpy out, build and apply of eight float64 images
        {"name": "regrid 64x64 s8", "kind": "regrid", "nx": 64, "ny": 64, "mx": 48, "my": 48, "stack": 8,
         "dtype": "float64"},
        # an image between an ordinary pair of odd, non-square grids that
        # are new to the program: their weights, applied once
        {"name": "build 333x257", "kind": "build", "nx": 333, "ny": 257, "mx": 250, "my": 193},
        # the same at the benchmark's size, the largest single build
        {"name": "build 2048x2048", "kind": "build", "nx": 2048, "ny": 2048, "mx": 1536, "my": 1536},
        # uneven new pairs built together, each applied to its image, as a
        # pipeline over many fields does
        {"name": "batch 16", "kind": "batch", "pairs": 16, "lo": 64, "hi": 512},
        # saved weights on the benchmark's deep float32 stack, float64 result
        {"name": "apply comp 2048x2048 s64", "kind": "apply", "nx": 2048, "ny": 2048, "mx": 1536, "my": 1536,
         "stack": 64, "dtype": "float32", "accumulate": "compensated"},
        # a served request: odd sides, a few float32 slices, float32 result
        {"name": "apply fast 777x611 s8", "kind": "apply", "nx": 777, "ny": 611, "mx": 583, "my": 458,
         "stack": 8, "dtype": "float32", "accumulate": "fast"},
        # the default accumulation on float64 arrays (numpy's default type)
        {"name": "apply exact 1024x1024 s8", "kind": "apply", "nx": 1024, "ny": 1024, "mx": 768, "my": 768,
         "stack": 8, "dtype": "float64", "accumulate": "exact"},
        # one optimisation step on the output coordinates and the values
        {"name": "grad 512x512 s16", "kind": "grad", "nx": 512, "ny": 512, "mx": 384, "my": 384, "stack": 16,
         "dtype": "float32"},
        # one wavelength solution applied to a large set of spectra
        {"name": "rows 4096 x65536", "kind": "rows", "n": 4096, "m": 4096, "stack": 65536},
        # spectra that each have their own wavelength grid, numpy in and out
        {"name": "spectra 256 x512", "kind": "spectra", "count": 256, "n": 512, "m": 384},
        # the cells that hold the vertices of another grid
        {"name": "locate 1024x1024", "kind": "locate", "nx": 1024, "ny": 1024, "mx": 769, "my": 769},
        # holes in a few detector images, numpy in and out
        {"name": "fill 4x480x641", "kind": "fill", "stack": 4, "nx": 480, "ny": 641, "dtype": "float64",
         "iterations": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    nx, ny = _log_int(rng, lo, hi), _log_int(rng, lo, hi)
    ratio = rng.uniform(0.5, 1.25)
    return {"nx": nx, "ny": ny, "mx": max(2, round(ratio * nx)), "my": max(2, round(ratio * ny))}


def draw(rng):
    kind = rng.choice(("regrid", "build", "batch", "apply", "apply", "apply", "grad", "rows", "spectra", "locate",
                       "fill"))
    if kind == "regrid":
        return {"kind": kind, **_sides(rng, 16, 128), "stack": _log_int(rng, 1, 16),
                "dtype": rng.choice(("float32", "float64"))}
    if kind == "build":
        return {"kind": kind, **_sides(rng, 64, 1600)}
    if kind == "batch":
        return {"kind": kind, "pairs": rng.randint(4, 20), "lo": 32, "hi": _log_int(rng, 96, 512)}
    if kind == "apply":
        mode = rng.choice(("fast", "compensated", "exact"))
        return {"kind": kind, **_sides(rng, 64, 1600), "stack": _log_int(rng, 1, 64),
                "dtype": rng.choice(("float32", "float64")) if mode == "exact" else "float32", "accumulate": mode}
    if kind == "grad":
        return {"kind": kind, **_sides(rng, 64, 512), "stack": _log_int(rng, 1, 16),
                "dtype": rng.choice(("float32", "float64"))}
    if kind == "rows":
        return {"kind": kind, "n": _log_int(rng, 256, 4096), "m": _log_int(rng, 256, 4096),
                "stack": _log_int(rng, 512, 65536)}
    if kind == "spectra":
        return {"kind": kind, "count": _log_int(rng, 16, 512), "n": _log_int(rng, 64, 1024),
                "m": _log_int(rng, 64, 1024)}
    if kind == "locate":
        return {"kind": kind, **_sides(rng, 64, 1600)}
    return {"kind": kind, "stack": _log_int(rng, 1, 16), "nx": _log_int(rng, 64, 768), "ny": _log_int(rng, 64, 768),
            "dtype": rng.choice(("float32", "float64")), "iterations": 100}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------


def _distorted(nx, ny, angle, amp):
    """``(nx + 1) x (ny + 1)`` vertices on [-1, 1]^2, rotated, then bent."""
    x, y = torch.meshgrid(torch.linspace(-1, 1, nx + 1, dtype=F64, device="cuda"),
                          torch.linspace(-1, 1, ny + 1, dtype=F64, device="cuda"), indexing="ij")
    xr = x * math.cos(angle) - y * math.sin(angle)
    yr = x * math.sin(angle) + y * math.cos(angle)
    xr = xr + amp * torch.sin(math.pi * yr)
    yr = yr + amp * torch.sin(math.pi * xr)
    return xr, yr


def _rectilinear(mx, my, extent, jitter, gen):
    x, y = torch.meshgrid(torch.linspace(-extent, extent, mx + 1, dtype=F64, device="cuda"),
                          torch.linspace(-extent, extent, my + 1, dtype=F64, device="cuda"), indexing="ij")
    noise = torch.randn(2, mx + 1, my + 1, dtype=F64, device="cuda", generator=gen) * jitter
    return x + noise[0], y + noise[1]


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _pair(rng, gen, nx, ny, mx, my, jitter=2e-9):
    gi = _distorted(nx, ny, rng.uniform(0, 0.5), rng.uniform(0, 0.03))
    return gi, _rectilinear(mx, my, rng.uniform(0.9, 1.1), jitter, gen)


def _grids(case, seed):
    """The pair of a case and the generators after it."""
    rng, gen = np.random.default_rng(seed), _generator(seed)
    if case["kind"] == "grad":
        # learnable output coordinates: an unrotated input, jitter of about a
        # fortieth of a cell, as the differentiable workload starts from
        gi = _distorted(case["nx"], case["ny"], 0.0, 0.02)
        side = max(case["mx"], case["my"])
        go = _rectilinear(case["mx"], case["my"], 0.95, 0.0768 / side, gen)
    else:
        gi, go = _pair(rng, gen, case["nx"], case["ny"], case["mx"], case["my"])
    return gi, go, rng, gen


def _stack(case, gen, cells):
    """Log-normal(3, 1) brightness values."""
    v = torch.randn(case["stack"], cells, device="cuda", generator=gen).add_(3.0).exp_()
    return v.to(getattr(torch, case["dtype"]))


def _image(gen, grid):
    cells = (grid[0].shape[0] - 1) * (grid[0].shape[1] - 1)
    return torch.randn(1, cells, dtype=F64, device="cuda", generator=gen).add_(3.0).exp_()


def _batch_pairs(case, seed):
    rng, gen = np.random.default_rng(seed), _generator(seed)
    # the sides are the case's own, so that passes on other seeds cost the same
    sides = np.random.default_rng(case["pairs"] * 10007 + case["hi"])
    pairs = []
    for _ in range(case["pairs"]):
        nx, ny = (int(round(math.exp(sides.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(2))
        pairs.append(_pair(rng, gen, nx, ny, max(2, round(0.75 * nx)), max(2, round(0.75 * ny))))
    return pairs


def _rows_inputs(case, seed):
    gen = _generator(seed)
    rng = np.random.default_rng(seed)
    x = np.sort(rng.uniform(0, 1, case["n"]))
    p = np.linspace(x[0], x[-1], case["m"])
    v = torch.randn(case["stack"], case["n"], device="cuda", generator=gen).add_(3.0).exp_()
    return x, p, v


def _spectra_inputs(case, seed):
    """Per-spectrum edges: a dispersion relation with its own shift and
    curvature, onto another grid inside and outside of it."""
    rng = np.random.default_rng(seed)
    c, n, m = case["count"], case["n"], case["m"]
    u = np.linspace(0, 1, n + 1)
    x = u + rng.uniform(-0.05, 0.05, (c, 1)) + rng.uniform(-0.2, 0.2, (c, 1)) * u * (1 - u)
    y = np.linspace(-0.02, 1.02, m + 1) + rng.uniform(-0.02, 0.02, (c, 1))
    return x, y, rng.poisson(100, (c, n)).astype(np.float64)


def _fill_inputs(case, seed):
    """Smooth images with rectangular holes over about 8 % of the cells."""
    rng = np.random.default_rng(seed)
    t, nx, ny = case["stack"], case["nx"], case["ny"]
    x, y = np.meshgrid(np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    a = np.empty((t, nx, ny), dtype=case["dtype"])
    for k in range(t):
        fx, fy, ph = rng.uniform(1, 5), rng.uniform(1, 5), rng.uniform(0, 6)
        a[k] = 100 + 30 * np.sin(fx * x + ph) * np.cos(fy * y)
        holes, want = 0, 0.08 * nx * ny
        while holes < want:
            h, w = rng.integers(1, max(2, nx // 10)), rng.integers(1, max(2, ny // 10))
            i, j = rng.integers(0, nx - h + 1), rng.integers(0, ny - w + 1)
            a[k, i:i + h, j:j + w] = np.nan
            holes += h * w
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        pairs = _batch_pairs(case, seed)
        gen = _generator(seed + 1)
        return {"case": case, "pairs": pairs, "values": [_image(gen, gi) for gi, _ in pairs]}
    if kind == "rows":
        x, p, v = _rows_inputs(case, seed)
        w, shape_in, shape_out = rg.weights((x,), (p,), method="multilinear")
        ii, oo, vv = w[()]
        dw = rg.DeviceWeights.from_coo(ii, oo, vv, shape_in[0], shape_out[0])
        return {"case": case, "weights": dw, "values": v}
    if kind == "spectra":
        x, y, v = _spectra_inputs(case, seed)
        return {"case": case, "x": x, "y": y, "values": v}
    if kind == "fill":
        return {"case": case, "values": _fill_inputs(case, seed)}
    gi, go, rng, gen = _grids(case, seed)
    state = {"case": case, "in": gi, "out": go}
    if kind == "regrid":
        state["in"], state["out"] = (tuple(a.cpu().numpy() for a in g) for g in (gi, go))
        v = rng.poisson(100, (case["stack"], case["nx"], case["ny"]))
        state["values"] = v.astype(case["dtype"])
    elif kind == "build":
        state["values"] = _image(gen, gi)
    elif kind == "apply":
        state["weights"] = rg.build_conservative_2d(gi, go)
        state["values"] = _stack(case, gen, case["nx"] * case["ny"])
    elif kind == "grad":
        cells = case["nx"] * case["ny"]
        state["values"] = _stack(case, gen, cells).reshape(-1, case["nx"], case["ny"]).requires_grad_()
        # targets of the output's own size: cells hold integrals
        scale = cells / (case["mx"] * case["my"])
        state["target"] = scale * _stack(case, gen, case["mx"] * case["my"]).reshape(-1, case["mx"], case["my"])
        for g in go:
            g.requires_grad_()
    elif kind == "locate":
        state["points"] = tuple(g.reshape(-1) for g in go)
    return state


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "regrid":
        return rg.regrid(state["in"], state["out"], state["values"], axis_input=(-2, -1), axis_output=(-2, -1),
                         method="conservative")
    if kind == "build":
        return rg.build_conservative_2d(state["in"], state["out"]).apply(state["values"])
    if kind == "batch":
        return [w.apply(v) for w, v in zip(batching.build_batch(state["pairs"]), state["values"])]
    if kind == "apply" or kind == "rows":
        return state["weights"].apply(state["values"], accumulate=case.get("accumulate", "fast"))
    if kind == "grad":
        xo, yo = state["out"]
        out = autograd.regrid_conservative_2d(state["values"], state["in"], state["out"])
        loss = 0.5 * (out - state["target"]).square().sum()
        gv, gx, gy = torch.autograd.grad(loss, (state["values"], xo, yo))
        return {"out": out, "grad_values": gv, "grad_x": gx, "grad_y": gy}
    if kind == "spectra":
        return rg.regrid((state["x"],), (state["y"],), state["values"], axis_input=-1, axis_output=-1,
                         method="conservative")
    if kind == "locate":
        return rg.locate_2d(state["in"], *state["points"])
    return rg.fill(state["values"], axis=(-2, -1), num_iterations=case["iterations"])


# --------------------------------------------------------------------------
# bytes and operations a pass cannot do without
# --------------------------------------------------------------------------


def _entries(nx, ny, mx, my):
    """About the number of overlapping cell pairs of two such grids: the
    cells of both and the crossings of their lines."""
    return (nx + mx) * (ny + my)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sides = np.random.default_rng(case["pairs"] * 10007 + case["hi"])
        nbytes = flops = 0
        for _ in range(case["pairs"]):
            nx, ny = (int(round(math.exp(sides.uniform(math.log(case["lo"]), math.log(case["hi"])))))
                      for _ in range(2))
            w = work({"kind": "build", "nx": nx, "ny": ny, "mx": max(2, round(0.75 * nx)),
                      "my": max(2, round(0.75 * ny))})
            nbytes, flops = nbytes + w["bytes"], flops + w["flops"]
        return {"bytes": nbytes, "flops": flops}
    if kind == "rows":
        return {"bytes": 4 * case["stack"] * (case["n"] + case["m"]) + 24 * case["m"],
                "flops": 4 * case["stack"] * case["m"]}
    if kind == "spectra":
        n, m = case["n"], case["m"]
        return {"bytes": 8 * case["count"] * (2 * n + 2 * m), "flops": 4 * case["count"] * (n + m)}
    if kind == "fill":
        cells = case["stack"] * case["nx"] * case["ny"]
        return {"bytes": 2 * cells * np.dtype(case["dtype"]).itemsize, "flops": 0.08 * cells * 6 * case["iterations"]}
    nx, ny, mx, my = case["nx"], case["ny"], case["mx"], case["my"]
    vertices = 16 * ((nx + 1) * (ny + 1) + (mx + 1) * (my + 1))
    nnz = _entries(nx, ny, mx, my)
    if kind == "locate":
        return {"bytes": vertices + 16 * (mx + 1) * (my + 1), "flops": 40 * (mx + 1) * (my + 1)}
    if kind == "build":
        # every overlap polygon has about four edges, whose crossing and
        # area term take about 20 operations
        return {"bytes": vertices + 8 * (nx * ny + mx * my) + 12 * nnz, "flops": 82 * nnz}
    width = np.dtype(case["dtype"]).itemsize
    wide = 4 if case.get("accumulate") == "fast" or (kind == "grad" and width == 4) else 8
    stack = case["stack"]
    arrays = stack * (nx * ny * width + mx * my * wide)
    if kind == "apply":
        return {"bytes": arrays + nnz * (4 + wide) + 8 * mx * my, "flops": 2 * nnz * stack}
    if kind == "regrid":
        return {"bytes": vertices + arrays, "flops": (80 + 2 * stack) * nnz}
    # values, output, target, both gradients; forward, transposed, dL/dw and the areas' adjoint
    return {"bytes": 2 * vertices + 2 * arrays + stack * mx * my * width, "flops": (80 + 40 + 6 * stack) * nnz}


# --------------------------------------------------------------------------
# the same in 64 bits, without the package
# --------------------------------------------------------------------------


def _quads(x, y):
    q = [(slice(None, -1), slice(None, -1)), (slice(1, None), slice(None, -1)), (slice(1, None), slice(1, None)),
         (slice(None, -1), slice(1, None))]
    return torch.stack([x[s].reshape(-1) for s in q], 1), torch.stack([y[s].reshape(-1) for s in q], 1)


def _cross(ax, ay, bx, by):
    return ax * by - ay * bx


def _clipped(ax, ay, bx, by, qx, qy):
    """Twice the contour area of the edges' parts inside the convex,
    counter-clockwise quads."""
    dx, dy = bx - ax, by - ay
    t0, t1 = torch.zeros_like(ax), torch.ones_like(ax)
    for f in range(4):
        g = (f + 1) % 4
        sx, sy = qx[:, g] - qx[:, f], qy[:, g] - qy[:, f]
        at_a = _cross(sx, sy, ax - qx[:, f], ay - qy[:, f])
        step = _cross(sx, sy, dx, dy)
        safe = torch.where(step == 0, torch.ones_like(step), step)
        t = -at_a / safe
        t0 = torch.where(step > 0, torch.maximum(t0, t), t0)
        t1 = torch.where(step < 0, torch.minimum(t1, t), t1)
        t1 = torch.where((step == 0) & (at_a < 0), torch.full_like(t1, -1.0), t1)
    return torch.where(t1 > t0, (t1 - t0) * _cross(ax, ay, dx, dy), torch.zeros_like(t0))


def _overlap(ix, iy, ox, oy):
    """Overlap areas of pairs of convex quads over the area of the first."""
    x0, y0 = ix[:, :1].detach(), iy[:, :1].detach()
    ix, iy, ox, oy = ix - x0, iy - y0, ox - x0, oy - y0
    area2 = _cross(ix[:, 2] - ix[:, 0], iy[:, 2] - iy[:, 0], ix[:, 3] - ix[:, 1], iy[:, 3] - iy[:, 1])
    both = 0
    for e in range(4):
        f = (e + 1) % 4
        both = both + _clipped(ox[:, e], oy[:, e], ox[:, f], oy[:, f], ix, iy)
        both = both + _clipped(ix[:, e], iy[:, e], ix[:, f], iy[:, f], ox, oy)
    return both / area2


def _candidates(gi, go, lo, hi):
    """Pairs of input cells lo..hi and output cells whose boxes touch; the
    output grid is rectilinear but for its jitter."""
    qx, qy = _quads(*gi)
    qx, qy = qx[lo:hi], qy[lo:hi]
    first, last = [], []
    for q, v, axis in ((qx, go[0].detach(), 1), (qy, go[1].detach(), 0)):
        n = v.shape[1 - axis] - 1
        upper, lower = v.amax(axis)[1:].contiguous(), v.amin(axis)[:-1].contiguous()
        first.append(torch.searchsorted(upper, q.amin(1).contiguous(), right=True).clamp(0, n))
        last.append(torch.searchsorted(lower, q.amax(1).contiguous()).clamp(0, n))
    na, nb = ((b - a).clamp(min=0) for a, b in zip(first, last))
    count = na * nb
    cell = torch.repeat_interleave(torch.arange(count.numel(), device="cuda"), count)
    k = torch.arange(cell.numel(), device="cuda") - (torch.cumsum(count, 0) - count)[cell]
    a = first[0][cell] + k // nb[cell]
    b = first[1][cell] + k % nb[cell]
    return cell, a * (go[0].shape[1] - 1) + b, qx, qy


def _weights(gi, go):
    """(input cell, output cell, weight) of every overlapping pair."""
    ox, oy = _quads(*go)
    parts = []
    cells = (gi[0].shape[0] - 1) * (gi[0].shape[1] - 1)
    for lo in range(0, cells, 1 << 20):
        cell, out, qx, qy = _candidates(gi, go, lo, min(cells, lo + (1 << 20)))
        w = _overlap(qx[cell], qy[cell], ox[out], oy[out])
        keep = w != 0
        parts.append((cell[keep] + lo, out[keep], w[keep]))
    return tuple(torch.cat(p) for p in zip(*parts))


def _applied(entries, values, cells_out):
    ii, oo, ww = entries
    out = torch.zeros(values.shape[0], cells_out, dtype=F64, device="cuda")
    for d in range(values.shape[0]):
        out[d].index_add_(0, oo, ww * values[d].to(F64)[ii])
    return out


def _exact_grad(case, seed):
    gi, go, _, gen = _grids(case, seed)
    cells_in, cells_out = case["nx"] * case["ny"], case["mx"] * case["my"]
    values = _stack(case, gen, cells_in).to(F64)
    target = (cells_in / cells_out) * _stack(case, gen, cells_out)
    target = target.to(F64)
    ii, oo, ww = _weights(gi, go)
    out = _applied((ii, oo, ww), values, cells_out)
    grad = out - target
    g_values = _applied((oo, ii, ww), grad, cells_in)
    g_weight = torch.zeros_like(ww)
    for d in range(values.shape[0]):
        g_weight += grad[d][oo] * values[d][ii]
    xo, yo = (g.detach().requires_grad_() for g in go)
    qx, qy = _quads(*gi)
    gx, gy = torch.zeros_like(xo), torch.zeros_like(yo)
    for lo in range(0, ii.numel(), 1 << 20):
        s = slice(lo, lo + (1 << 20))
        ox, oy = _quads(xo, yo)
        part = (_overlap(qx[ii[s]], qy[ii[s]], ox[oo[s]], oy[oo[s]]) * g_weight[s]).sum()
        a, b = torch.autograd.grad(part, (xo, yo))
        gx, gy = gx + a, gy + b
    return {"out": out.reshape(-1, case["mx"], case["my"]),
            "grad_values": g_values.reshape(-1, case["nx"], case["ny"]), "grad_x": gx, "grad_y": gy}


def _exact_fill(case, seed):
    a = torch.from_numpy(_fill_inputs(case, seed)).cuda().to(F64)
    hole = torch.isnan(a)
    # numpy's median: the mean of the two middle values
    guess = torch.tensor([float(np.nanmedian(s)) for s in a.cpu().numpy()], dtype=F64, device="cuda")
    a = torch.where(hole, guess[:, None, None], a)
    nx, ny = case["nx"], case["ny"]
    i, j = torch.meshgrid(torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda"), indexing="ij")
    seam = torch.zeros_like(i)
    if nx % 2:
        seam = seam + (i == nx - 1)
    if ny % 2:
        seam = seam + (j == ny - 1)
    cx, cy = ((n - 1) ** 2 / 4.0 for n in (nx, ny))
    for _ in range(case["iterations"]):
        for colour in range(2):
            # odd periodic axes join cells of one colour: those come last
            for phase in range(int(seam.max()) + 1):
                at = hole & ((i + j) % 2 == colour) & (seam == phase)
                new = (cx * (a.roll(1, 1) + a.roll(-1, 1)) + cy * (a.roll(1, 2) + a.roll(-1, 2))) / (2 * (cx + cy))
                a = torch.where(at, new, a)
    return a


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        gen = _generator(seed + 1)
        return [_applied(_weights(gi, go), _image(gen, gi), (go[0].shape[0] - 1) * (go[0].shape[1] - 1))
                for gi, go in _batch_pairs(case, seed)]
    if kind == "locate":
        return None  # whole numbers
    if kind == "fill":
        return _exact_fill(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "rows":
        x, p, v = _rows_inputs(case, seed)
        i = np.clip(np.searchsorted(x, p, side="right") - 1, 0, case["n"] - 2)
        t = torch.from_numpy((p - x[i]) / (x[i + 1] - x[i])).cuda()
        i = torch.from_numpy(i).cuda()
        out = torch.empty(case["stack"], case["m"], dtype=F64, device="cuda")
        for d in range(0, case["stack"], 4096):
            s = v[d:d + 4096]
            out[d:d + 4096] = s[:, i].to(F64) * (1 - t) + s[:, i + 1].to(F64) * t
        return out
    if kind == "spectra":
        x, y, v = _spectra_inputs(case, seed)
        out = np.empty((case["count"], case["m"]))
        for k in range(case["count"]):
            level = v[k].mean()
            density = (v[k] - level)
            total = np.concatenate([[0.0], np.cumsum(density)])
            part = np.interp(y[k], x[k], total)
            index = np.interp(y[k], x[k], np.arange(case["n"] + 1.0))
            out[k] = np.diff(part) + level * np.diff(index)
        return out
    gi, go, rng, gen = _grids(case, seed)
    if kind == "regrid":
        values = torch.from_numpy(rng.poisson(100, (case["stack"], case["nx"], case["ny"]))).cuda()
        values = values.to(F64).reshape(case["stack"], -1)
        # the default perturbation of the output grid
        rng = np.random.default_rng(42)
        go = [g.cpu().numpy() for g in go]
        go = tuple(torch.from_numpy(rng.normal(g, np.ptp(g) * 1e-9)).cuda() for g in go)
        out = _applied(_weights(gi, go), values, case["mx"] * case["my"])
        return out.reshape(-1, case["mx"], case["my"])
    values = _image(gen, gi) if kind == "build" else _stack(case, gen, case["nx"] * case["ny"])
    return _applied(_weights(gi, go), values, case["mx"] * case["my"])
