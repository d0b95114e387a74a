"""Level by level in one CTA, x in a ring: entries whose column left the ring
long ago, among them infinite ones."""
import numpy as np
import pytest

from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["order", "multirow"])
def test_infinite_entries_far_back(torch_cuda, mode):
    torch = torch_cuda
    import sptrsv_b200 as S

    n, at = 40000, {30000: (5, np.inf), 36001: (700, -np.inf), 39990: (12, 0.5)}
    rows = [[(i - 1, -0.5)] if i % 16 else [] for i in range(n)]  # a chain, cut now and then
    for i in range(16, n, 16):
        rows[i] = [(i - 9, 0.25)]
    for i, e in at.items():
        rows[i] = [e] + rows[i]
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.array([c for i, r in enumerate(rows) for c in [q for q, _ in r] + [i]], dtype=np.int32)
    va = np.array([v for r in rows for v in [w for _, w in r] + [1.0]])
    m = gen.from_arrays(rp, ci, va)
    b = np.random.default_rng(1).uniform(1, 2, n)
    x = b.copy()
    with np.errstate(invalid="ignore"):
        for i, r in enumerate(rows):
            for c, v in r:
                x[i] -= v * x[c]
    assert np.isinf(x).any() and np.isinf(x[30000])
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(n, n, m.nnz, *(a.data_ptr() for a in t))
    info = S.AnalysisInfo()
    info.mode = S.ALL
    assert S.run_analysis(info, L) == 0
    got = torch.empty(n, dtype=torch.float64, device="cuda")
    call = S.csr_L_solve_order if mode == "order" else S.csr_L_solve_multirow
    call(L, info, torch.from_numpy(b).cuda(), got, n)
    S.sync_status()
    got = got.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(x))
    assert np.array_equal(np.where(np.isinf(got), got, 0), np.where(np.isinf(x), x, 0))
    fin = np.isfinite(x)
    assert np.allclose(got[fin], x[fin], rtol=1e-11, atol=1e-11)
    S.free_device_analysis(None, info)
