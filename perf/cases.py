"""Timed cases of the solver: what a program that uses it has it do, through
its public entry points, over the range of matrices it is made for.

A case is a dict of plain values:
  call     which entry point a pass goes through
             host      run_solver: host b in, host x out (the drop-in interface)
             dropin    csr_L_solve_{simple,order,multirow} on device vectors
             plan      Plan.solve_f64 / Plan.solve_ir
             batch     Batch.solve: many systems, one launch
             analysis  run_analysis on a device CSR
  matrix   banded | grid2d | grid3d | zipf | blockdiag, with its sizes
  other options are described at `prepare`.

Matrices follow the generators of the library (same shapes and
distributions), made on the GPU from the seed: strictly lower entries in
ascending column order, the diagonal last in every row, row diagonally
dominant.  b = L x_true.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

import sptrsv_b200 as S
from sptrsv_b200 import select
from sptrsv_b200.batch import Batch

DEV = "cuda"


# ------------------------------------------------------------------- cases
def listed():
    return [
        # The reference's own test driver: analyse a small system once, then
        # solve host vectors through run_solver.  Latency and fixed costs.
        {"name": "host_small", "call": "host", "solver": "multirow", "matrix": "banded", "n": 5000, "bandwidth": 64,
         "off_lo": 4, "off_hi": 8},
        # A small stencil solved again and again inside an outer iteration
        # (a preconditioner), FP32 + FP64 refinement, the plan as created.
        {"name": "plan_small_ir", "call": "plan", "solve": "ir", "schedule": "default", "nrhs": 1, "matrix": "grid2d",
         "nx": 61, "ny": 47},
        # The drop-in solvers of the reference on device vectors: the long
        # chain (2D Laplacian), the narrow band, and independent dense blocks
        # solved without any analysis.
        {"name": "dropin_multirow_grid", "call": "dropin", "solver": "multirow", "matrix": "grid2d", "nx": 2048,
         "ny": 2048},
        {"name": "dropin_order_banded", "call": "dropin", "solver": "order", "matrix": "banded", "n": 100_000,
         "bandwidth": 256, "off_lo": 8, "off_hi": 8},
        {"name": "dropin_simple_blocks", "call": "dropin", "solver": "simple", "matrix": "blockdiag", "n": 300_007,
         "block": 32},
        # Plans whose schedule the shipped selector picks: the benchmark's
        # banded and grid systems, a ragged 3D stencil refined from FP32, and
        # the wide shallow DAG.
        {"name": "plan_banded", "call": "plan", "solve": "f64", "schedule": "select", "nrhs": 1, "matrix": "banded",
         "n": 100_000, "bandwidth": 256, "off_lo": 8, "off_hi": 8},
        {"name": "plan_grid", "call": "plan", "solve": "f64", "schedule": "select", "nrhs": 1, "matrix": "grid2d",
         "nx": 2048, "ny": 2048},
        {"name": "plan_grid3d_ir", "call": "plan", "solve": "ir", "schedule": "select", "nrhs": 1, "matrix": "grid3d",
         "nx": 101, "ny": 90, "nz": 97},
        {"name": "plan_zipf", "call": "plan", "solve": "f64", "schedule": "select", "nrhs": 1, "matrix": "zipf",
         "n": 2_000_000, "max_off": 256},
        # The same DAG with a block of right-hand sides.
        {"name": "plan_zipf_k16", "call": "plan", "solve": "f64", "schedule": "default", "nrhs": 16, "matrix": "zipf",
         "n": 2_000_000, "max_off": 256},
        # Many systems of uneven size, 1-32 right-hand sides each, in one launch.
        {"name": "batch_512", "call": "batch", "systems": 512, "n_lo": 1000, "n_hi": 200_000, "bw_lo": 16,
         "bw_hi": 4096, "off_lo": 4, "off_hi": 16, "k_max": 32, "precision": 64, "block_rows": 0},
        # The analysis every one of them starts from, on a stencil of a domain
        # with holes (each coupling is there with probability `keep`).
        {"name": "analysis_grid", "call": "analysis", "matrix": "grid2d", "nx": 1023, "ny": 1025, "keep": 0.98},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, n_lo, n_hi, kinds):
    kind = rng.choice(kinds)
    n = _log(rng, n_lo, n_hi)
    if kind == "banded":
        lo = rng.randint(4, 8)
        return {"matrix": kind, "n": min(n, 400_000), "bandwidth": _log(rng, 16, 4096), "off_lo": lo,
                "off_hi": rng.randint(lo, 16)}
    if kind == "grid2d":
        nx = max(8, int(round(math.sqrt(n) * math.exp(rng.uniform(-0.5, 0.5)))))
        return {"matrix": kind, "nx": nx, "ny": max(8, n // nx)}
    if kind == "grid3d":
        nx = max(4, int(round(n ** (1 / 3) * math.exp(rng.uniform(-0.3, 0.3)))))
        ny = max(4, int(round(n ** (1 / 3) * math.exp(rng.uniform(-0.3, 0.3)))))
        return {"matrix": kind, "nx": nx, "ny": ny, "nz": max(4, n // (nx * ny))}
    if kind == "zipf":
        return {"matrix": kind, "n": n, "max_off": 256}
    return {"matrix": "blockdiag", "n": min(n, 1_000_000), "block": 32}


def draw(rng):
    call = rng.choice(["host", "dropin", "dropin", "plan", "plan", "plan", "mrhs", "batch", "analysis"])
    every = ["banded", "grid2d", "grid3d", "zipf", "blockdiag"]
    if call == "host":
        return {"call": "host", "solver": rng.choice(["order", "multirow"]), **_matrix(rng, 1000, 200_000, every)}
    if call == "dropin":
        solver = rng.choice(["simple", "order", "multirow"])
        return {"call": "dropin", "solver": solver, **_matrix(rng, 1000, 500_000 if solver == "simple" else 2_000_000,
                                                              every)}
    if call == "plan":
        return {"call": "plan", "solve": rng.choice(["f64", "f64", "ir"]), "schedule": rng.choice(["default", "select"]),
                "nrhs": 1, **_matrix(rng, 1000, 2_000_000, every)}
    if call == "mrhs":
        return {"call": "plan", "solve": "f64", "schedule": "default", "nrhs": rng.randint(2, 32),
                **_matrix(rng, 1000, 1_000_000, every)}
    if call == "batch":
        return {"call": "batch", "systems": _log(rng, 4, 128), "n_lo": 1000, "n_hi": _log(rng, 2000, 200_000),
                "bw_lo": 16, "bw_hi": _log(rng, 64, 4096), "off_lo": 4, "off_hi": 16, "k_max": _log(rng, 1, 32),
                "precision": rng.choice([32, 64]), "block_rows": rng.choice([0, 0, 4096])}
    return {"call": "analysis", "keep": round(rng.uniform(0.9, 0.99), 3), **_matrix(rng, 1000, 2_000_000, every)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _row_sums(data, rowptr):
    return torch.segment_reduce(data, "sum", offsets=rowptr.long(), initial=0.0)


def _csr(cols, g, diag, lo, hi, part=1.0):
    """CSR from per-row candidate columns [n, k] (ascending, -1 where there is
    none), off-diagonals U(lo, hi), the diagonal last: `diag`, or
    1 + sum |off-diagonals| of the row when it is None.  part < 1: each
    candidate is there with that probability only."""
    n = cols.shape[0]
    if part < 1.0:
        cols = torch.where(_rand(g, cols.numel()).view(cols.shape) < part, cols, -1)
    rows = torch.arange(n, device=DEV, dtype=cols.dtype)
    full = torch.cat([cols, rows[:, None]], 1)
    keep = full >= 0
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = keep.sum(1).cumsum(0)
    col = full[keep].int()
    return _values(rowptr, col, g, diag, lo, hi)


def _values(rowptr, col, g, diag, lo, hi):
    val = lo + (hi - lo) * _rand(g, col.numel())
    last = rowptr[1:].long() - 1
    if diag is None:
        val[last] = 0.0
        val[last] = 1.0 + _row_sums(val.abs(), rowptr)
    else:
        val[last] = diag
    return rowptr, col, val


def _banded_cols(local, width, count, g):
    """Per row, `count` distinct columns uniform in the `width` rows before it
    (Floyd's sampling, one step per column for all rows at once), ascending."""
    kmax = int(count.max())
    n = local.numel()
    picked = torch.full((n, kmax), -1, dtype=torch.int32, device=DEV)
    for j in range(kmax):
        live = j < count
        top = (width - count + j).clamp(min=0)  # t uniform in [0, top]
        t = (_rand(g, n) * (top + 1)).floor().int().minimum(top)
        again = (picked[:, :j] == t[:, None]).any(1) if j else torch.zeros(n, dtype=torch.bool, device=DEV)
        picked[:, j] = torch.where(live, torch.where(again, top, t), -1)
    off = torch.where(picked >= 0, local[:, None] - 1 - picked, -1)
    return off.sort(1).values


def _banded(local, bandwidth, lo, hi, g):
    """local: row index inside its system; bandwidth: per row."""
    want = (lo + (_rand(g, local.numel()) * (hi - lo + 1)).floor().int()).clamp(max=hi)
    width = torch.minimum(local, bandwidth)
    return _banded_cols(local, width, torch.minimum(want, width), g)


def _matrix_of(case, g):
    kind, part = case["matrix"], case.get("keep", 1.0)
    if kind == "banded":
        local = torch.arange(case["n"], device=DEV, dtype=torch.int32)
        bw = torch.full_like(local, case["bandwidth"])
        return _csr(_banded(local, bw, case["off_lo"], case["off_hi"], g), g, None, -1.0, 1.0, part)
    if kind == "grid2d":
        nx, ny = case["nx"], case["ny"]
        i = torch.arange(nx * ny, device=DEV, dtype=torch.int32)
        cols = torch.stack([torch.where(i >= nx, i - nx, -1), torch.where(i % nx > 0, i - 1, -1)], 1)
        return _csr(cols, g, 4.0, -1.1, -0.9, part)
    if kind == "grid3d":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        i = torch.arange(nx * ny * nz, device=DEV, dtype=torch.int32)
        cols = torch.stack([torch.where(i >= nx * ny, i - nx * ny, -1), torch.where((i // nx) % ny > 0, i - nx, -1),
                            torch.where(i % nx > 0, i - 1, -1)], 1)
        return _csr(cols, g, 6.0, -1.1, -0.9, part)
    if kind == "blockdiag":
        n, w = case["n"], case["block"]
        i = torch.arange(n, device=DEV, dtype=torch.int32)
        j = torch.arange(w - 1, device=DEV, dtype=torch.int32)
        cols = torch.where(j[None, :] < (i % w)[:, None], (i - i % w)[:, None] + j[None, :], -1)
        return _csr(cols, g, None, -1.0, 1.0, part)
    n, cap = case["n"], case["max_off"]
    z = np.arange(1, cap + 1, dtype=np.float64) ** -1.5
    cdf = torch.from_numpy(np.cumsum(z) / 2.6123753486854883).to(DEV)  # P(Z <= z) = sum z^-s / zeta(1.5)
    row = torch.arange(n, device=DEV, dtype=torch.int64)
    count = torch.searchsorted(cdf, _rand(g, n)).clamp(max=cap).minimum(row)
    rows = torch.repeat_interleave(row, count)
    cols = (_rand(g, rows.numel()) * rows).floor().long().minimum(rows - 1)
    key = torch.unique(torch.cat([rows * n + cols, row * n + row]))
    rows, col = key // n, (key % n).int()
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = torch.bincount(rows, minlength=n).cumsum(0)
    return _values(rowptr, col, g, None, -1.0, 1.0)


def _matvec(m, x):
    """L x, row by row; x is n or n x k."""
    rowptr, col, val = m
    if x.dim() == 1:
        return _row_sums(val * x[col.long()], rowptr)
    return torch.stack([_row_sums(val * c[col.long()], rowptr) for c in x.T.contiguous()], 1).contiguous()


def _sp_mat(m):
    rowptr, col, val = m
    n = rowptr.numel() - 1
    return S.SpMat(n, n, col.numel(), rowptr.data_ptr(), col.data_ptr(), val.data_ptr())


def _inputs(case, seed):
    """(matrix, b) of a single-system case."""
    g = _generator(seed)
    m = _matrix_of(case, g)
    n, k = m[0].numel() - 1, case.get("nrhs", 1)
    shape = n if k == 1 else (n, k)
    if case["matrix"] == "zipf":
        x = torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)
    else:
        x = 2 * torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) - 1
    return m, _matvec(m, x)


def _batch_sizes(case):
    """(rows, bandwidths, right-hand sides) of a batch's systems: rows and
    bandwidths log-uniform, right-hand sides uniform.  The case fixes them;
    the seed makes patterns and values."""
    rng = np.random.default_rng(case["systems"])
    ns = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), case["systems"])).astype(np.int64)
    bws = np.exp(rng.uniform(np.log(case["bw_lo"]), np.log(case["bw_hi"]), case["systems"])).astype(np.int32)
    return ns, bws, rng.integers(1, case["k_max"] + 1, case["systems"])


def _batch_inputs(case, seed):
    """(per-system matrices, right-hand side counts, per-system b)."""
    g = _generator(seed)
    ns, bws, ks = _batch_sizes(case)
    mats, bs, s = [], [], 0
    while s < len(ns):  # systems made together, up to 4 M rows at a time
        e = s + 1
        while e < len(ns) and ns[s:e + 1].sum() <= 4_000_000:
            e += 1
        count = torch.from_numpy(ns[s:e]).to(DEV)
        first = count.cumsum(0) - count
        row = torch.arange(int(ns[s:e].sum()), device=DEV)
        local = (row - torch.repeat_interleave(first, count)).int()
        bw = torch.repeat_interleave(torch.from_numpy(bws[s:e]).to(DEV), count)
        rowptr, col, val = _csr(_banded(local, bw, case["off_lo"], case["off_hi"], g), g, None, -1.0, 1.0)
        at = rowptr[torch.cat([first, count.sum()[None]])].tolist()  # entries before each system
        start = first.tolist()
        for j in range(e - s):
            n = int(ns[s + j])
            rp = (rowptr[start[j]:start[j] + n + 1] - at[j]).contiguous()
            # columns are already local to the system; the diagonal is its row of the group
            c = col[at[j]:at[j + 1]].clone()
            c[rp[1:].long() - 1] -= start[j]
            m = (rp, c, val[at[j]:at[j + 1]].clone())
            x = 2 * torch.rand(n, int(ks[s + j]), generator=g, device=DEV, dtype=torch.float64) - 1
            mats.append(m)
            bs.append(_row_sums(m[2][:, None] * x[m[1].long()], rp))
        s = e
    return mats, [int(k) for k in ks], bs


# ------------------------------------------------------- what a program keeps
class _Analysed:
    """A device CSR with its analysis; both end with this object."""

    def __init__(self, m, mode):
        self.m = m  # keeps the device arrays alive
        self.L = _sp_mat(m)
        self.info = None
        if mode != S.SIMPLE:
            self.info = S.AnalysisInfo()
            self.info.mode = mode
            S.run_analysis(self.info, self.L)

    def __del__(self):
        if self.info is not None:
            S.free_device_analysis(None, self.info)


_MODES = {"simple": S.SIMPLE, "order": S.ORDER, "multirow": S.MULTIROW}
_selector = None


def _shipped_selector():
    global _selector
    if _selector is None:
        _selector = select.Mlp.load(Path(select.__file__).with_name("selector_weights.npz"))
    return _selector


class _Ints:
    """A device int32 array of the library, as torch reads foreign memory."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    """solver: the drop-in solver (host, dropin).  solve: f64, or ir (FP32 with
    FP64 refinement).  schedule: the plan's default, or what the shipped
    selector picks.  precision, block_rows: Batch.solve / set_partition."""
    if case["call"] == "batch":
        mats, ks, bs = _batch_inputs(case, seed)
        torch.cuda.synchronize()
        batch = Batch([_sp_mat(m) for m in mats], ks)
        if case["block_rows"]:
            batch.set_partition(case["block_rows"])
        b = torch.cat([v.reshape(-1) for v in bs])
        return {"case": case, "batch": batch, "b": b, "x": torch.empty_like(b)}
    m, b = _inputs(case, seed)
    torch.cuda.synchronize()
    state = {"case": case}
    if case["call"] == "analysis":
        state["A"] = _Analysed(m, S.SIMPLE)
        state["A"].info = S.AnalysisInfo()
        state["A"].info.mode = S.ALL
        n = state["A"].L.nr  # at most one warp per row
        state["out"] = {k: torch.empty(n + 1, dtype=torch.int32, device=DEV)
                        for k in ("iorder", "inv_iorder", "lev_size", "ibase_row", "ivect_size_warp", "warp_lev")}
        return state
    if case["call"] == "plan":
        A = _Analysed(m, S.ALL)
        plan = S.Plan(A.L, A.info)
        if case["schedule"] == "select":
            _shipped_selector().select(plan, A.L, A.info)
        state.update(A=A, plan=plan, b=b, x=torch.empty_like(b))
        return state
    state["A"] = _Analysed(m, _MODES[case["solver"]])
    if case["call"] == "host":
        state.update(b=b.cpu().numpy(), x=np.empty(b.numel()))
    else:
        state.update(b=b, x=torch.empty_like(b))
    return state


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "batch":
        state["batch"].solve(state["b"], state["x"], precision=case["precision"])
        return state["x"]
    A = state["A"]
    if call == "plan":
        solve = state["plan"].solve_ir if case["solve"] == "ir" else state["plan"].solve_f64
        solve(state["b"], state["x"], nrhs=case["nrhs"])
        return state["x"]
    n = A.L.nr
    if call == "host":
        S.run_solver(A.L, A.info, state["b"], state["x"], n)
        return state["x"]
    if call == "dropin":
        if case["solver"] == "simple":
            S.csr_L_solve_simple(A.L, state["b"], state["x"], n)
        elif case["solver"] == "order":
            S.csr_L_solve_order(A.L, A.info, state["b"], state["x"], n)
        else:
            S.csr_L_solve_multirow(A.L, A.info, state["b"], state["x"], n)
        return state["x"]
    S.run_analysis(A.info, A.L)
    # copies, as the next analysis into the same struct releases these arrays;
    # the ones whose length the pattern decides end in -1
    info = A.info
    arrays = {"iorder": (info.iorder, n), "inv_iorder": (info.inv_iorder, n), "lev_size": (info.lev_size, info.nlevs),
              "ibase_row": (info.ibase_row, info.n_warps + 1), "ivect_size_warp": (info.ivect_size_warp, info.n_warps),
              "warp_lev": (info.warp_lev, info.n_warps)}
    for k, (ptr, count) in arrays.items():
        state["out"][k][:count] = torch.as_tensor(_Ints(ptr, count), device=DEV)
        state["out"][k][count:] = -1
    return state["out"]


# ------------------------------------------------------------- what it needs
def _sizes(case):
    """(rows, expected entries) of a single-system case."""
    kind = case["matrix"]
    if kind == "banded":
        n = case["n"]
        off = n * min((case["off_lo"] + case["off_hi"]) / 2, case["bandwidth"])
    elif kind == "grid2d":
        nx, ny = case["nx"], case["ny"]
        n, off = nx * ny, 2 * nx * ny - nx - ny
    elif kind == "grid3d":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n, off = nx * ny * nz, 3 * nx * ny * nz - nx * ny - ny * nz - nx * nz
    elif kind == "blockdiag":
        n = case["n"]
        off = n * (case["block"] - 1) / 2
    else:
        n, cap = case["n"], case["max_off"]
        z = np.arange(1, cap + 1, dtype=np.float64)
        p = z ** -1.5 / 2.6123753486854883
        off = n * float((p * (z - 1)).sum() + cap * (1 - p.sum()))
    return n, n + case.get("keep", 1.0) * off


def work(case):
    if case["call"] == "batch":
        # int32 row pointers and columns, f64 values, b in and x out
        ns, _, ks = _batch_sizes(case)
        nnz = ns * (1 + (case["off_lo"] + case["off_hi"]) / 2)
        return {"bytes": float((4 * ns + 12 * nnz + 16 * ns * ks).sum()), "flops": float((2 * nnz * ks).sum())}
    n, nnz = _sizes(case)
    if case["call"] == "analysis":  # the pattern in; orders and the warp map out
        return {"bytes": 4 * n + 4 * nnz + 8 * n, "flops": nnz}
    k = case.get("nrhs", 1)
    return {"bytes": 4 * (n + 1) + 12 * nnz + 16 * n * k, "flops": 2 * nnz * k}


# -------------------------------------------------------------------- exact
def _substitute(m, b):
    """L^-1 b in 64 bits by sweeps x <- (b - (L - D) x) / D, repeated until
    nothing changes: after as many sweeps as L has levels every row holds its
    forward substitution, with the row's products added in column order."""
    rowptr, col, val = m
    last = rowptr[1:].long() - 1
    d = val[last].clone()
    off = val.clone()
    off[last] = 0.0
    x = b / (d if b.dim() == 1 else d[:, None])
    at = col.long()
    for sweep in range(1, 200_000):
        if b.dim() == 1:
            new = (b - _row_sums(off * x[at], rowptr)) / d
        else:
            new = (b - _row_sums(off[:, None] * x[at], rowptr)) / d[:, None]
        if sweep % 16 == 0 and torch.equal(new, x):
            break
        x = new
    return x


def exact(case, seed):
    if case["call"] == "batch":
        mats, ks, bs = _batch_inputs(case, seed)
        return torch.cat([_substitute(m, b).reshape(-1) for m, b in zip(mats, bs)])
    m, b = _inputs(case, seed)
    if case["call"] == "analysis":
        return None  # whole numbers
    if b.dim() == 1:
        x = _substitute(m, b)
    else:  # a few columns at a time
        x = torch.cat([_substitute(m, c.contiguous()) for c in b.split(4, 1)], 1)
    return x.cpu().numpy() if case["call"] == "host" else x
