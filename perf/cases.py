"""Representative calls of the RL / RLZ transform framework, with their sizes.

Each case is one call (or one pair of calls) a program makes through the public
Python mirror: ``spectralTransform!`` / ``gridTransform!`` on RL and RLZ grids
in FP64 and in FP32 with the refined spline solve, a batch of uneven RL grids, a
patch chain and the regular-grid output.  ``listed`` holds fixed sizes (the
shapes of the repository's benchmark and tests, and odd ones between them),
``draw`` random ones of the same ranges.

``exact`` restates the transforms with dense torch FP64 operations: spline
projection and solve as matrices, the rings through ``torch.fft``, the Chebyshev
columns as cosine matrices.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "springsteel.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import springsteel_gpu as S  # noqa: E402

ZMAX = 20000.0


def _rl(name, call, cells, nvars, precision, kmax=-1, bc="natural"):
    return {"name": name, "geometry": "RL", "call": call, "cells": cells, "vars": nvars, "precision": precision,
            "kmax": kmax, "bc": bc, "levels": 1, "low_pass": -1}


def _rlz(name, call, cells, levels, nvars, precision, kmax=-1, bc="natural", low_pass=-1):
    return {"name": name, "geometry": "RLZ", "call": call, "cells": cells, "levels": levels, "vars": nvars,
            "precision": precision, "kmax": kmax, "bc": bc, "low_pass": low_pass}


def listed():
    return [
        # the smallest grid of the tests' range: one step of a unit test or a toy vortex; launches count
        _rl("rl24_f64_round", "round", 24, 1, "f64"),
        # the 100-cell single-variable vortex grid every RL user starts from
        _rl("rl100_f64_round", "round", 100, 1, "f64"),
        # a shallow-water step on a fine RL grid: several variables, odd ring counts, binary32
        _rl("rl251_f32_round", "round", 251, 4, "f32", bc="dirichlet"),
        # a small 3-D case with a wavenumber cap, a spectral filter and odd sizes
        _rlz("rlz37_f64_round", "round", 37, 21, 3, "f64", kmax=72, bc="neumann", low_pass=60),
        # a mid-size binary32 step: 3 variables, an odd number of levels
        _rlz("rlz125_f32_round", "round", 125, 45, 3, "f32"),
        # the headline grid (200 cells, 32 levels, 5 variables, FP64), each direction
        _rlz("rlz200_f64_forward", "forward", 200, 32, 5, "f64"),
        _rlz("rlz200_f64_inverse", "inverse", 200, 32, 5, "f64"),
        # the large binary32 grid (400 cells, 64 levels), four of its variables, each direction
        _rlz("rlz400_f32_forward", "forward", 400, 64, 4, "f32"),
        _rlz("rlz400_f32_inverse", "inverse", 400, 64, 4, "f32"),
        # independent uneven RL grids of an ensemble, one fused batch replayed as a graph
        {"name": "batch10_rl_f32", "geometry": "RL", "call": "batch", "grids": 10, "cells_min": 50, "cells_max": 400,
         "vars_max": 4, "precision": "f32"},
        # a 3-patch RLZ chain (40/120/40 cells, 2:1 interfaces): multiGridTransform!
        {"name": "chain_rlz_f64", "geometry": "RLZ", "call": "chain", "cells": 40, "levels": 24, "vars": 2,
         "precision": "f64"},
        # output step of a model: every field on the regular (r, λ, z) lattice, into host memory
        {"name": "regular_rlz60_f64", "geometry": "RLZ", "call": "regular", "cells": 60, "levels": 24, "vars": 2,
         "precision": "f64", "kmax": -1, "bc": "natural", "low_pass": -1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rl", "rl", "rlz", "rlz", "rlz", "rlz", "other"])
    precision = rng.choice(["f64", "f32"])
    if kind == "rl":
        cells = _log_int(rng, 10, 400)
        kmax = -1 if rng.random() < 0.7 else rng.randint(4, 3 * cells)
        c = _rl("", rng.choice(["forward", "inverse", "round"]), cells, rng.randint(1, 5), precision, kmax,
                rng.choice(["natural", "dirichlet", "neumann"]))
    elif kind == "rlz":
        cells = _log_int(rng, 12, 200 if precision == "f64" else 400)
        levels = rng.randint(8, 40 if precision == "f64" else 64)
        # no more work than the largest listed grid of the same precision
        most = (200 ** 2 * 32 * 5 if precision == "f64" else 400 ** 2 * 64 * 4) / (cells ** 2 * levels)
        call = rng.choice(["forward", "inverse", "round"])
        nvars = rng.randint(1, max(1, min(6, int(most / 2 if call == "round" else most))))
        kmax = -1 if rng.random() < 0.7 else rng.randint(4, 3 * cells)
        low = -1 if rng.random() < 0.7 else rng.randint(3, 2 * cells)
        c = _rlz("", call, cells, levels, nvars, precision, kmax, rng.choice(["natural", "dirichlet", "neumann"]), low)
    else:
        call = rng.choice(["batch", "chain", "regular"])
        if call == "batch":
            lo = rng.randint(20, 120)
            c = {"geometry": "RL", "call": call, "grids": rng.randint(2, 10), "cells_min": lo,
                 "cells_max": lo + rng.randint(10, 280), "vars_max": rng.randint(1, 4), "precision": precision}
        elif call == "chain":
            c = {"geometry": "RLZ", "call": call, "cells": rng.randint(8, 40), "levels": rng.randint(8, 24),
                 "vars": rng.randint(1, 2), "precision": "f64"}
        else:
            c = {"geometry": "RLZ", "call": call, "cells": rng.randint(10, 60), "levels": rng.randint(8, 24),
                 "vars": rng.randint(1, 2), "precision": "f64", "kmax": -1, "bc": "natural", "low_pass": -1}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ parameters
def _bcs(name):
    return {"natural": (S.NaturalBC(), S.NaturalBC()), "dirichlet": (S.NaturalBC(), S.DirichletBC()),
            "neumann": (S.NeumannBC(), S.NeumannBC())}[name]


def _params(case, cells=None, nvars=None):
    cells = case["cells"] if cells is None else cells
    nvars = case["vars"] if nvars is None else nvars
    left, right = _bcs(case.get("bc", "natural"))
    kw = dict(geometry=case["geometry"], iMin=0.0, iMax=float(cells), num_cells=cells,
              vars={"v%d" % i: i for i in range(1, nvars + 1)}, BCL={"default": left}, BCR={"default": right},
              precision=case["precision"], max_wavenumber={"default": case.get("kmax", -1)})
    if case["geometry"] == "RLZ":
        kw.update(kMin=0.0, kMax=ZMAX, kDim=case["levels"], BCB={"default": S.DirichletBC()},
                  BCT={"default": S.DirichletBC()})
    if case.get("low_pass", -1) >= 0:
        kw["fourier_filter"] = {"default": S.SpectralFilter(low_pass=case["low_pass"], window="exponential",
                                                            taper_width=8)}
    return S.SpringsteelGridParameters(**kw)


class _View:
    """Device memory of a grid for ``torch.as_tensor``; a tensor of it keeps the grid alive."""

    def __init__(self, grid, ptr, shape, size):
        self.grid = grid
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f%d" % size, "data": (ptr, False), "version": 3,
                                         "strides": None}


def _physical(grid):
    """grid.physical on the device as (nslots, nvars, points), no copy."""
    d = grid.dims
    first = grid.device_array("physical", 0, 1)
    return torch.as_tensor(_View(grid, first.data_ptr(), (d["nslots"], d["nvars"], d["n_physical"]),
                                 first.element_size()), device="cuda")


def _spectral(grid):
    """grid.spectral on the device as (nvars, coefficients), no copy."""
    d = grid.dims
    first = grid.device_array("spectral", 0)
    return torch.as_tensor(_View(grid, first.data_ptr(), (d["nvars"], d["n_spectral"]), first.element_size()),
                           device="cuda")


# ------------------------------------------------------------------ inputs
def _ring_points(gp):
    """(r, λ) of every ring point, on the device."""
    rings = torch.arange(1, gp.iDim + 1, device="cuda") + gp.patchOffsetL
    L = 4 + 4 * rings
    ring = torch.repeat_interleave(torch.arange(gp.iDim, device="cuda"), L)
    l_of = torch.arange(int(L.sum()), device="cuda") - torch.repeat_interleave(torch.cumsum(L, 0) - L, L)
    dx = (gp.iMax - gp.iMin) / gp.num_cells
    q = torch.tensor([0.5 - 0.5 * math.sqrt(0.6), 0.5, 0.5 + 0.5 * math.sqrt(0.6)], dtype=torch.float64, device="cuda")
    mish = (gp.iMin + (torch.arange(gp.num_cells, device="cuda", dtype=torch.float64)[:, None] + q) * dx).reshape(-1)
    dl = 2 * math.pi / L.double()
    lam = (0.5 * dl * (rings - 1))[ring] + dl[ring] * l_of
    return mish[ring], lam


def _levels(n):
    return ZMAX * 0.5 * (1 - torch.cos(torch.arange(n, dtype=torch.float64, device="cuda") * math.pi / (n - 1)))


def _fields(gp, seed):
    """(nvars, points): each variable a sum of 8 seeded Gaussian vortex blobs plus noise."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    r, lam = _ring_points(gp)
    x, y = r * torch.cos(lam), r * torch.sin(lam)
    dtype = torch.float32 if gp.precision == "f32" else torch.float64
    levels = gp.kDim if gp.geometry == "RLZ" else 1
    z = _levels(levels) if levels > 1 else None
    out = torch.empty((len(gp.vars), r.numel() * levels), dtype=dtype, device="cuda")
    for v in range(len(gp.vars)):
        plan, column = [], []
        for _ in range(8):
            rc, tc = gp.iMax * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
            w, amp, zc = rng.uniform(5, 30), rng.normal(), rng.uniform(0, ZMAX)
            plan.append(amp * torch.exp(-((x - rc * math.cos(tc)) ** 2 + (y - rc * math.sin(tc)) ** 2) / w ** 2))
            if z is not None:
                column.append(torch.exp(-(((z - zc) / (100 * w)) ** 2)))
        f = torch.stack(plan, 1)
        f = f.sum(1) if z is None else f.to(dtype) @ torch.stack(column, 0).to(dtype)
        out[v] = f.reshape(-1).to(dtype)
        out[v] += 1e-3 * torch.randn(out.shape[1], generator=gen, device="cuda", dtype=dtype)
    return out


def _coefficients(gp, seed):
    """(nvars, n_spectral) B-vectors of a model state: smooth in r, falling in wavenumber and level."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    dtype = torch.float32 if gp.precision == "f32" else torch.float64
    K, b = gp.iDim + gp.patchOffsetL, gp.b_iDim
    bk = gp.b_kDim if gp.geometry == "RLZ" else 1
    k = torch.arange(1, K + 1, device="cuda", dtype=torch.float64)
    fall = torch.cat([torch.ones(1, device="cuda", dtype=torch.float64),
                      torch.repeat_interleave(1.0 / (1.0 + (k / 6.0) ** 2), 2)])
    deep = 1.0 / (1.0 + (torch.arange(bk, device="cuda", dtype=torch.float64) / 4.0) ** 2)
    m = torch.arange(b, device="cuda", dtype=torch.float64)
    out = torch.empty((len(gp.vars), bk, 1 + 2 * K, b), dtype=dtype, device="cuda")
    for v in range(len(gp.vars)):
        shapes = torch.stack([torch.exp(-(((m - rng.uniform(0, b)) / rng.uniform(4, 4 + b / 6)) ** 2))
                              for _ in range(6)]).to(dtype)
        mix = torch.randn((bk, 1 + 2 * K, 6), generator=gen, device="cuda", dtype=dtype)
        mix *= (deep[:, None, None] * fall[None, :, None]).to(dtype)
        out[v] = mix @ shapes
    return out.reshape(len(gp.vars), -1)


# ------------------------------------------------------------------ prepare / run
def _batch_shapes(case):
    rng = random.Random("%d %d %d" % (case["grids"], case["cells_min"], case["cells_max"]))
    return [(rng.randint(case["cells_min"], case["cells_max"]), rng.randint(1, case["vars_max"]))
            for _ in range(case["grids"])]


def _chain_params(case):
    c = case["cells"]
    return S.chain_grid_params([0.0, float(c), 2.5 * c, 3.5 * c], [c, 3 * c, c], geometry="RLZ", kMin=0.0, kMax=ZMAX,
                               kDim=case["levels"], BCB={"default": S.DirichletBC()}, BCT={"default": S.DirichletBC()},
                               vars={"v%d" % i: i for i in range(1, case["vars"] + 1)}, precision=case["precision"])


def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        grids = [S.createGrid(_params(case, c, v)) for c, v in _batch_shapes(case)]
        for i, g in enumerate(grids):
            _physical(g)[0].copy_(_fields(g.params, seed * 100 + i))
        torch.cuda.synchronize()
        batch = S.Batch(grids)
        return {"call": call, "grids": grids, "batch": batch,
                "out": [[_spectral(g)] + list(_physical(g)) for g in grids]}
    if call == "chain":
        grids = [S.createGrid(p) for p in _chain_params(case)]
        for i, g in enumerate(grids):
            _spectral(g).copy_(_coefficients(g.params, seed * 100 + i))
        torch.cuda.synchronize()
        return {"call": call, "chain": S.PatchChain(grids), "out": [list(_physical(g)) for g in grids]}
    gp = _params(case)
    grid = S.createGrid(gp)
    if call in ("inverse", "regular"):
        _spectral(grid).copy_(_coefficients(gp, seed))
    else:
        _physical(grid)[0].copy_(_fields(gp, seed))
    torch.cuda.synchronize()
    state = {"call": call, "grid": grid}
    if call == "forward":
        state["out"] = _spectral(grid)
    elif call == "inverse":
        state["out"] = list(_physical(grid))
    elif call == "round":
        state["out"] = [_spectral(grid)] + list(_physical(grid))
    else:
        state["axes"] = S.regular_axes(gp)
    return state


def run(state):
    call = state["call"]
    if call in ("forward", "round"):
        S.spectralTransform_b(state["grid"])
    if call in ("inverse", "round"):
        S.gridTransform_b(state["grid"])
    if call == "batch":
        state["batch"].run(what=3)
    if call == "chain":
        state["chain"].multiGridTransform()
    if call == "regular":
        return S.regularGridTransform(state["grid"], *state["axes"])
    return state["out"]


# ------------------------------------------------------------------ work
def _grid_work(gp, forward, inverse):
    es = 4 if gp.precision == "f32" else 8
    rlz = gp.geometry == "RLZ"
    nv, kz, bk = len(gp.vars), gp.kDim if rlz else 1, gp.b_kDim if rlz else 1
    L = 4.0 + 4.0 * (np.arange(1, gp.iDim + 1) + gp.patchOffsetL)
    points, nspec = L.sum(), bk * (1 + 2 * (gp.iDim + gp.patchOffsetL)) * gp.b_iDim
    ring = nv * bk * float((2.5 * L * np.log2(L)).sum())
    column = nv * points * 2.5 * 2 * (kz - 1) * math.log2(2 * (kz - 1)) if kz > 2 else 0.0
    rows = nv * bk * float((L / 2 - 1).sum())
    bytes_ = flops = 0.0
    if forward:
        bytes_ += es * nv * (points * kz + nspec)
        flops += column + ring + 24.0 * nv * nspec
    if inverse:
        bytes_ += es * nv * (points * kz * (7 if rlz else 5) + nspec)
        flops += 7 * column + 5 * ring + 16.0 * nv * nspec + 24.0 * rows
    return bytes_, flops


def work(case):
    call = case["call"]
    if call == "batch":
        parts = [_grid_work(_params(case, c, v), True, True) for c, v in _batch_shapes(case)]
    elif call == "chain":
        parts = [_grid_work(p, False, True) for p in _chain_params(case)]
    elif call == "regular":
        gp = _params(case)
        r, lam, z = S.regular_axes(gp)
        points, K = len(r) * len(lam) * len(z), gp.iDim
        spec = gp.b_kDim * (1 + 2 * K) * gp.b_iDim
        # per radius and level the ring coefficients, then a 2K-term sum per point and ring variant
        parts = [(8.0 * len(gp.vars) * (spec + 7 * points),
                  len(gp.vars) * (24.0 * len(r) * gp.b_kDim * (1 + 2 * K) + 7 * points * 2.5 * math.log2(len(lam))))]
    else:
        parts = [_grid_work(_params(case), call != "inverse", call != "forward")]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ------------------------------------------------------------------ exact values
_GAMMA = {"natural": None, "dirichlet": (-4.0, -1.0), "neumann": (0.0, 1.0)}


def _bspline(x, m, xmin, dx, d):
    """Cubic B-spline φ_m and derivatives (Ooyama 2002) at x[:, None], nodes m[None, :]."""
    delta = (x[:, None] - (xmin + m[None, :] * dx)) / dx
    z = delta.abs()
    one = (z < 1).double()
    two = (z < 2).double()
    sgn = torch.where(delta > 0, -1.0, 1.0)
    if d == 0:
        return two * ((2 - z) ** 3 / 6 - one * (1 - z) ** 3 * (4 / 6))
    if d == 1:
        return two * ((2 - z) ** 2 / 6 - one * (1 - z) ** 2 * (4 / 6)) * sgn * 3 / dx
    if d == 2:
        return two * ((2 - z) - one * (1 - z) * 4) / dx ** 2
    return two * torch.where(z > 1, 1.0, torch.where(z < 1, -3.0, 0.0)) * sgn / dx ** 3


def _spline(gp, left, right):
    """(SB, SA, [SI, SIx, SIxx]) as dense FP64 matrices."""
    n, b = gp.num_cells, gp.b_iDim
    dx = (gp.iMax - gp.iMin) / n
    q = torch.tensor([0.5 - 0.5 * math.sqrt(0.6), 0.5, 0.5 + 0.5 * math.sqrt(0.6)], dtype=torch.float64, device="cuda")
    w = torch.tensor([5 / 18, 8 / 18, 5 / 18], dtype=torch.float64, device="cuda").repeat(n) * dx
    x = (gp.iMin + (torch.arange(n, device="cuda", dtype=torch.float64)[:, None] + q) * dx).reshape(-1)
    m = torch.arange(-1, n + 2, device="cuda", dtype=torch.float64)
    phi = [_bspline(x, m, gp.iMin, dx, d) for d in range(4)]
    eps = (2.0 * dx / (2 * math.pi)) ** 6
    PQ = phi[0].T @ (w[:, None] * phi[0]) + eps * (phi[3].T @ (w[:, None] * phi[3]))
    rank_l, rank_r = int(left is not None), int(right is not None)
    fold = torch.zeros((b - rank_l - rank_r, b), dtype=torch.float64, device="cuda")
    idx = torch.arange(fold.shape[0], device="cuda")
    fold[idx, idx + rank_l] = 1.0
    if left is not None:
        fold[0, 0], fold[1, 0] = left
    if right is not None:
        fold[-1, -1], fold[-2, -1] = right
    solve = fold.T @ torch.linalg.inv(fold @ PQ @ fold.T) @ fold
    return phi[0].T * w[None, :], solve, phi[:3]


def _cheb(gp):
    """(forward bk × N, [inverse, d/dz, d²/dz²] N × bk) of columns with Dirichlet ends."""
    N, bk = gp.kDim, gp.b_kDim
    j = torch.arange(N, dtype=torch.float64, device="cuda")
    cos = torch.cos(torch.remainder(j[:, None] * j[None, :], 2 * (N - 1)) * (math.pi / (N - 1)))
    end = torch.full((N,), 2.0, dtype=torch.float64, device="cuda")
    end[0] = end[-1] = 1.0
    fwd = cos * end[None, :] / (2 * (N - 1))
    if bk == N:
        fwd = fwd * torch.exp(-36.0 * ((j + 1) / N) ** 36)[:, None]
    inv = cos * end[None, :]
    alt = torch.where(j % 2 == 0, 1.0, -1.0).double()
    gamma = torch.eye(N, dtype=torch.float64, device="cuda")[:, :bk]
    gamma = gamma + torch.ones_like(j)[:, None] * (end * -0.5 / (N - 1))[None, :bk]
    gamma = gamma + alt[:, None] * (-alt / (N - 1) * end * 0.5)[None, :bk]
    D = torch.triu(2.0 * j[None, :].expand(N, N), 1) * (torch.remainder(j[None, :] - j[:, None], 2) == 1)
    D = D / (-0.5 * (gp.kMax - gp.kMin))
    return fwd[:bk], [inv @ gamma, inv @ D @ gamma, inv @ D @ (D @ gamma)]


def _rings(gp):
    jo = 0
    for r in range(gp.iDim):
        ri = r + 1 + gp.patchOffsetL
        L = 4 + 4 * ri
        kmax = ri if gp.shared_ring_kmax() < 0 else min(ri, gp.shared_ring_kmax())
        k = torch.arange(kmax + 1, device="cuda", dtype=torch.float64)
        phase = torch.exp(1j * (k * (0.5 * (2 * math.pi / L) * (ri - 1))))
        yield r, L, kmax, k, phase, jo
        jo += L


def _exact_forward(gp, case, phys):
    """phys: (points, levels) FP64 of one variable -> (bk, 1 + 2K, b) coefficients."""
    K = gp.iDim + gp.patchOffsetL
    g = _GAMMA[case["bc"]]
    SB, _, _ = _spline(gp, g if case["bc"] == "neumann" else None, g)
    C = phys @ _cheb(gp)[0].T if gp.geometry == "RLZ" else phys
    F = torch.zeros((gp.iDim, C.shape[1], 1 + 2 * K), dtype=torch.float64, device="cuda")
    for r, L, kmax, k, phase, jo in _rings(gp):
        X = torch.fft.rfft(C[jo:jo + L].T, norm="forward")[:, :kmax + 1] * phase.conj()
        F[r, :, 0] = X[:, 0].real
        F[r, :, 1:2 * kmax:2] = X[:, 1:].real
        F[r, :, 2:2 * kmax + 1:2] = X[:, 1:].imag
    spec = (SB @ F.reshape(gp.iDim, -1)).reshape(gp.b_iDim, C.shape[1], 1 + 2 * K).permute(1, 2, 0).contiguous()
    if case["low_pass"] >= 0:
        k = torch.div(torch.arange(1 + 2 * K, device="cuda") + 1, 2, rounding_mode="floor")
        over = (k - case["low_pass"]).double()
        wgt = torch.where(over <= 0, 1.0, torch.where(over > 8, 0.0, torch.exp(-4.0 * (over / 8) ** 2)))
        spec *= wgt[None, :, None]
    return spec


def _exact_inverse(gp, case, spec):
    """spec: (bk, 1 + 2K, b) FP64 of one variable -> list of physical slots, each (points × levels,)."""
    g = _GAMMA[case["bc"]]
    _, solve, SI = _spline(gp, g if case["bc"] == "neumann" else None, g)
    rlz = gp.geometry == "RLZ"
    cols = _cheb(gp)[1] if rlz else None
    bk, ns, b = spec.shape
    points = sum(4 + 4 * (r + 1 + gp.patchOffsetL) for r in range(gp.iDim))
    a = spec.reshape(-1, b) @ solve.T
    slots = [None] * (7 if rlz else 5)
    for d, wants in enumerate((((0, 0), (1, 3), (2, 4)), ((0, 1),), ((0, 2),))):
        u = (a @ SI[d].T).reshape(bk, ns, gp.iDim)
        for order, slot in wants:
            H = torch.empty((points, bk), dtype=torch.float64, device="cuda")
            for r, L, kmax, k, phase, jo in _rings(gp):
                X = torch.zeros((bk, L // 2 + 1), dtype=torch.complex128, device="cuda")
                X[:, 0] = u[:, 0, r]
                X[:, 1:kmax + 1] = torch.complex(u[:, 1:2 * kmax:2, r], u[:, 2:2 * kmax + 1:2, r])
                X[:, :kmax + 1] *= phase * (1j * k) ** order
                H[jo:jo + L] = torch.fft.irfft(X, n=L, norm="forward").T
            slots[slot] = (H @ cols[0].T if rlz else H).reshape(-1)
            if rlz and slot == 0:
                slots[5], slots[6] = ((H @ cols[i].T).reshape(-1) for i in (1, 2))
    return slots


def exact(case, seed):
    if case["call"] in ("batch", "chain", "regular"):
        return None
    gp = _params(case)
    call, nv = case["call"], case["vars"]
    levels = case["levels"] if case["geometry"] == "RLZ" else 1
    if call == "inverse":
        K = gp.iDim + gp.patchOffsetL
        spec = _coefficients(gp, seed)
        specs = [spec[v].double().reshape(-1, 1 + 2 * K, gp.b_iDim) for v in range(nv)]
        del spec
    else:
        f = _fields(gp, seed)
        specs = [_exact_forward(gp, case, f[v].double().reshape(-1, levels)) for v in range(nv)]
        del f
    if call == "forward":
        return torch.stack([s.reshape(-1) for s in specs])
    per_var = [_exact_inverse(gp, case, s) for s in specs]
    slots = []
    for i in range(len(per_var[0])):
        slots.append(torch.stack([p[i] for p in per_var]))
        for p in per_var:
            p[i] = None
    if call == "inverse":
        return slots
    return [torch.stack([s.reshape(-1) for s in specs])] + slots
