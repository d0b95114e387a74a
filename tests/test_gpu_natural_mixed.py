"""Natural-order solves of a warp that holds a row out of order behind its first
entries: rows that took a column of the warp while they waited must not take it
again when the warp goes on in the form for such rows."""
import ctypes

import numpy as np
import pytest

from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _matrix(front):
    """A chain of `front` rows, then warps of 32: rows 0 and 1 without columns, row
    5 long and out of order behind its fourth entry, hanging on the chain's end, row
    9 reading rows 0 and 5.  Whole numbers, so sums are exact in any order."""
    rows = [[i - 1] if i else [] for i in range(front)]
    for w in range(16):
        r0 = front + 32 * w
        warp = [[] for _ in range(32)]
        warp[5] = [front - 40, front - 30, front - 20, front - 1, r0 + 1, w]
        warp[9] = [r0, r0 + 5]
        warp[20] = [w + 3, r0, r0 + 9]
        rows += warp
    rng = np.random.default_rng(front)
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(list(r) + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = rng.choice([-1.0, 1.0], ci.size)
    va[rp[1:] - 1] = 1.0
    return gen.from_arrays(rp, ci, va), rng.integers(-9, 10, len(rows)).astype(np.float64)


@pytest.mark.parametrize("front", [4096, 20480])
def test_columns_taken_while_waiting_are_taken_once(torch_cuda, front):
    torch = torch_cuda
    import sptrsv_b200 as S
    from sptrsv_b200 import _lib

    m, xt = _matrix(front)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t))
    b = torch.from_numpy(m.matvec(xt)).cuda()
    x = torch.empty_like(b)
    for _ in range(3):
        x.fill_(float("nan"))
        S.csr_L_solve_simple(L, b, x, m.n)
        S.sync_status()
        assert np.array_equal(x.cpu().numpy(), xt)
        x.fill_(float("nan"))
        assert _lib.lib().sptrsv_solve_ir_noalloc(ctypes.byref(L), b.data_ptr(), x.data_ptr(), 0, None) == 0
        assert np.array_equal(x.cpu().numpy(), xt)
