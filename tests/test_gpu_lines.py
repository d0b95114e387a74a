"""Drop-in solves of stencils line by line: line lengths around the chunk of 32
and the CTA's lines, a ragged last line, dropped couplings, couplings into the
same line, forms that the rule does not take, values that must not be
multiplied up, infinities."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _stencil(nx, n, offs, seed=0, keep=1.0, off=None):
    """n rows on lines of nx, row (i, j) reads (i + a, j + b) of offs; dominant unless off is given."""
    rng = np.random.default_rng(seed)
    r = np.arange(n)
    i, j = r % nx, r // nx
    cols, rows = [r], [r]
    for a, b in offs:
        ok = (0 <= i + a) & (i + a < nx) & (0 <= j + b) & (rng.random(n) < keep)
        cols.append((j + b)[ok] * nx + (i + a)[ok])
        rows.append(r[ok])
    cols, rows = np.concatenate(cols), np.concatenate(rows)
    order = np.lexsort((cols, rows))
    ci, rows = cols[order].astype(np.int32), rows[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    last = rp[1:] - 1
    va = rng.uniform(-1, 1, ci.size) if off is None else np.full(ci.size, float(off))
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1]) if off is None else 1.0
    return gen.from_arrays(rp, ci, va)


FIVE, NINE = [(-1, 0), (0, -1)], [(-1, 0), (-1, -1), (0, -1), (1, -1)]
MATS = {
    **{f"five_{nx}": (lambda nx=nx: _stencil(nx, nx * 400 + 17, FIVE, seed=nx)) for nx in (32, 33, 64, 95, 96, 97, 300)},
    "long_lines": lambda: _stencil(3001, 3001 * 130 - 1, FIVE, seed=1),       # four lines a CTA
    "longer_lines": lambda: _stencil(8000, 8000 * 70, FIVE, seed=2),          # two
    "few_lines": lambda: _stencil(9000, 9000 * 3 + 5, FIVE, seed=3),
    "dropped": lambda: _stencil(257, 257 * 300, FIVE, seed=4, keep=0.9),
    "nine": lambda: _stencil(200, 200 * 300, NINE, seed=5),
    "seven_2d": lambda: _stencil(200, 200 * 300, FIVE + [(-1, -1)], seed=6),
    "two_lines_up": lambda: _stencil(150, 150 * 300, FIVE + [(0, -2), (1, -3)], seed=7),
    "same_line_40": lambda: _stencil(150, 150 * 300, FIVE + [(-40, 0)], seed=8),
    "same_line_3": lambda: _stencil(150, 150 * 300, FIVE + [(-3, 0)], seed=9),
    "six_off": lambda: _stencil(150, 150 * 300, NINE + [(0, -2), (0, -3)], seed=10),
    "grid3d": lambda: gen.grid3d(67, 43, 45, seed=11),
}


def _solve(S, torch, m, b, solvers=("multirow", "order")):
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t))
    info = S.AnalysisInfo()
    info.mode = S.ALL
    S.run_analysis(info, L)
    bd, out = torch.from_numpy(b).cuda(), []
    for s in solvers:
        x = torch.full_like(bd, float("nan"))
        (S.csr_L_solve_multirow if s == "multirow" else S.csr_L_solve_order)(L, info, bd, x, m.n)
        S.sync_status()
        out.append(x.cpu().numpy())
    S.free_device_analysis(None, info)
    return out


@pytest.mark.parametrize("name", list(MATS))
def test_lines_match_the_oracle(torch_cuda, name):
    import sptrsv_b200 as S

    m = MATS[name]()
    b = m.matvec(gen.vector(m.n, "uniform", seed=11))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    for got in _solve(S, torch_cuda, m, b):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


def test_lines_with_growing_factors_are_exact_in_whole_numbers(torch_cuda):
    """Factors of 2 along the line: no scan multiplies them; whole numbers below 2^53."""
    import sptrsv_b200 as S

    m = _stencil(150, 150 * 300, FIVE, off=-1)
    rows = np.repeat(np.arange(m.n), np.diff(m.rowptr))
    m.val[(m.colidx == rows - 1) & (rows % 2 == 0)] = -2.0
    xt = np.random.default_rng(3).integers(-9, 10, m.n).astype(np.float64)
    for got in _solve(S, torch_cuda, m, m.matvec(xt)):
        assert np.array_equal(got, xt)


@pytest.mark.parametrize("keep", [1.0, 0.8])
def test_lines_with_infinities(torch_cuda, keep):
    """The rows that depend on an infinite b, infinite or NaN as in a solve row by row; the
    ones beside them that do not (couplings are missing) stay finite."""
    import sptrsv_b200 as S

    m = _stencil(150, 150 * 300, FIVE, seed=12, keep=keep)
    off = np.ones(m.nnz, bool)
    off[m.rowptr[1:] - 1] = False
    m.val[off] = -1e-9
    b = m.matvec(gen.vector(m.n, "uniform", seed=1))
    b[[150 * 290 + 7]] = np.inf
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    fin = np.isfinite(ref)
    for got in _solve(S, torch_cuda, m, b):
        assert np.array_equal(got[~fin], ref[~fin], equal_nan=True)
        assert np.abs(got[fin] - ref[fin]).max() <= 1e-12 * np.abs(ref[fin]).max()
