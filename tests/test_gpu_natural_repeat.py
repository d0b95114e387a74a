"""Natural-order solves give the same bits on every run, whichever rows of a
warp came first."""
import ctypes

import numpy as np
import pytest

from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu

MATS = {
    "grid": lambda: gen.grid2d(333, 200, seed=1),
    "short_lines": lambda: gen.grid2d(7, 3001, seed=2),
    "grid3d": lambda: gen.grid3d(37, 30, 31, seed=3),
    "band": lambda: gen.banded(20000, 64, 4, 8, seed=4),
}


@pytest.mark.parametrize("name", list(MATS))
def test_the_same_bits_on_every_run(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S
    from sptrsv_b200 import _lib

    m = MATS[name]()
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t))
    b = torch.from_numpy(m.matvec(gen.vector(m.n, "uniform", seed=11))).cuda()
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(0, rows_per_warp=32, ir_max_iters=1)

    def noalloc(x):
        assert _lib.lib().sptrsv_solve_ir_noalloc(ctypes.byref(L), b.data_ptr(), x.data_ptr(), 1, None) == 0

    for solve in (lambda x: S.csr_L_solve_simple(L, b, x, m.n), lambda x: p.solve_f64(b, x), lambda x: p.solve_ir(b, x),
                  noalloc):
        first = None
        for _ in range(12):
            x = torch.full_like(b, float("nan"))
            solve(x)
            S.sync_status()
            got = x.cpu().numpy().view(np.int64)
            first = got if first is None else first
            assert np.array_equal(got, first)
    p.close()
    S.free_device_analysis(None, info)
