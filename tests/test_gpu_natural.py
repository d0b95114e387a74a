"""Solves in natural order (SIMPLE, the allocation-free solve): sizes around
the warp and the group, stencils whose lines start anywhere, rows longer than
a round, rows inside one warp, factors the scan does not take, infinities and
NaN, and device CSRs whose rows are not sorted."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _rows(rows, off=None, diag=None, seed=0):
    """CSR of these columns per row (in this order), diagonal last, dominant unless given."""
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(list(r) + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = rng.uniform(-1, 1, ci.size) if off is None else np.full(ci.size, float(off))
    last = rp[1:] - 1
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1]) if diag is None else diag
    return gen.from_arrays(rp, ci, va)


def _stencil27(nx, ny, nz):
    rows = []
    for k in range(nz):
        for j in range(ny):
            for i in range(nx):
                me = (k * ny + j) * nx + i
                r = [((k + c) * ny + j + b) * nx + i + a for c in (-1, 0) for b in (-1, 0, 1) for a in (-1, 0, 1)
                     if 0 <= k + c and 0 <= j + b < ny and 0 <= i + a < nx]
                rows.append([q for q in r if q < me])
    return _rows(rows)


MATS = {
    **{f"chain_{n}": (lambda n=n: _rows([[i - 1] if i else [] for i in range(n)], seed=n)) for n in (1, 31, 33, 256, 257)},
    **{f"grid_{nx}": (lambda nx=nx: gen.grid2d(nx, 61, seed=1)) for nx in (3, 31, 32, 33, 255, 300)},
    "grid3d": lambda: gen.grid3d(37, 12, 13, seed=3),
    "stencil27": lambda: _stencil27(11, 9, 8),
    "dense_band": lambda: gen.banded(1500, 20, 20, 20, seed=5),
    "band": lambda: gen.banded(5000, 64, 4, 8, seed=6),
    "wide_band": lambda: gen.banded(6001, 900, 0, 24, seed=7),
    "blocks_32": lambda: gen.blockdiag(1000, 32, seed=4),
    "blocks_48": lambda: gen.blockdiag(1003, 48, seed=4),
    "zipf": lambda: gen.zipf(20000, 1.5, 256, seed=2),
}


def _device(S, torch, m):
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    return S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t)), t


def _noalloc(L, b, x):
    from sptrsv_b200 import _lib

    assert _lib.lib().sptrsv_solve_ir_noalloc(ctypes.byref(L), b.data_ptr(), x.data_ptr(), 2, None) == 0


@pytest.mark.parametrize("name", list(MATS))
def test_natural_solves_match_the_oracle(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = MATS[name]()
    b = m.matvec(gen.vector(m.n, "uniform", seed=11))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    top = np.abs(ref).max()
    L, keep = _device(S, torch, m)
    bd = torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)

    def off():
        S.sync_status()
        return float(np.abs(x.cpu().numpy() - ref).max() / top)

    S.csr_L_solve_simple(L, bd, x, m.n)
    assert off() <= 1e-12
    x.fill_(float("nan"))
    _noalloc(L, bd, x)
    assert off() <= 1e-12
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(0, rows_per_warp=32, ir_max_iters=2)
    x.fill_(float("nan"))
    p.solve_f64(bd, x)
    assert off() <= 1e-12
    p.close()
    S.free_device_analysis(None, info)


def test_growing_chain_is_exact_in_whole_numbers(torch_cuda):
    """Factors of 2, which the scan does not take: whole numbers far below 2^53 throughout."""
    torch = torch_cuda
    import sptrsv_b200 as S

    m = _rows([[i - 1] if i % 40 else [] for i in range(700)], off=-2, diag=1.0)
    xt = np.random.default_rng(3).integers(-9, 10, m.n).astype(np.float64)
    L, keep = _device(S, torch, m)
    x = torch.empty(m.n, dtype=torch.float64, device="cuda")
    S.csr_L_solve_simple(L, torch.from_numpy(m.matvec(xt)).cuda(), x, m.n)
    S.sync_status()
    assert np.array_equal(x.cpu().numpy(), xt)


@pytest.mark.parametrize("order", ["descending", "shuffled"])
def test_rows_in_any_order(torch_cuda, order):
    torch = torch_cuda
    import sptrsv_b200 as S

    rng = np.random.default_rng(5)
    m = gen.banded(2000, 40, 3, 14, seed=9)
    ref = O.solve(m.rowptr, m.colidx, m.val, b := m.matvec(gen.vector(m.n, "uniform", seed=1)))
    ci, va = m.colidx.copy(), m.val.copy()
    for i in range(m.n):
        s, e = m.rowptr[i], m.rowptr[i + 1] - 1
        k = np.arange(s, e)[::-1] if order == "descending" else s + rng.permutation(e - s)
        ci[s:e], va[s:e] = m.colidx[k], m.val[k]
    L, keep = _device(S, torch, gen.from_arrays(m.rowptr, ci, va))
    bd = torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    S.csr_L_solve_simple(L, bd, x, m.n)
    S.sync_status()
    assert O.rel_err(x.cpu().numpy(), ref) <= 1e-12
    x.fill_(0)
    _noalloc(L, bd, x)
    assert O.rel_err(x.cpu().numpy(), ref) <= 1e-12


def test_infinities_and_nan_spread_as_in_substitution(torch_cuda):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = _rows([[c for c in (i - 40, i - 1) if c >= 0 and (c != i - 1 or i % 45)] for i in range(600)], off=1e-200, diag=1.0)
    b = np.ones(m.n)
    b[7], b[300] = np.inf, np.nan
    x = b.copy()
    for i in range(m.n):
        for k in range(m.rowptr[i], m.rowptr[i + 1] - 1):
            x[i] -= m.val[k] * x[m.colidx[k]]
    L, keep = _device(S, torch, m)
    got = torch.empty(m.n, dtype=torch.float64, device="cuda")
    S.csr_L_solve_simple(L, torch.from_numpy(b).cuda(), got, m.n)
    S.sync_status()
    got = got.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(x))
    assert np.array_equal(got[~np.isnan(x)], x[~np.isnan(x)])
