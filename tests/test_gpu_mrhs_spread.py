"""Many right-hand sides on long rows and wide levels, a row's entries shared out
over its lanes: row lengths around the round of 16, counts of right-hand sides
whose rows of x are whole 16-byte copies, and ones that are not."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _layers(widths, per_level, seed):
    """Levels of per_level rows; row i of a level reads widths[i % len] rows, one of them of the level before."""
    rng = np.random.default_rng(seed)
    rows, r = [], 0
    for lev in range(6):
        for i in range(per_level):
            k = widths[i % len(widths)] if lev else 0
            c = []
            if k:
                c = set(rng.integers(0, lev * per_level, k).tolist()) | {(lev - 1) * per_level + i}
            rows.append(sorted(c) + [r])
            r += 1
    rp = np.concatenate([[0], np.cumsum([len(q) for q in rows])])
    ci = np.concatenate(rows).astype(np.int32)
    va = rng.uniform(-1, 1, ci.size)
    last = rp[1:] - 1
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1])
    return gen.from_arrays(rp, ci, va)


@pytest.mark.parametrize("k", [9, 10, 12, 16, 17, 20, 31, 32])
def test_spread_rounds_match_the_oracle(torch_cuda, k):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = _layers([1, 2, 7, 14, 15, 16, 17, 31, 32, 33, 63, 100, 257], 1100, seed=k)
    assert m.nnz - m.n >= 8 * m.n and m.n >= 1024 * 6
    b = m.matvec(gen.vector(m.n * k, "uniform", seed=3), k)
    ref = O.solve(m.rowptr, m.colidx, m.val, b, nrhs=k)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t))
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    bd = torch.from_numpy(b).cuda()
    x = torch.full_like(bd, float("nan"))
    top = np.abs(ref).max()
    for _ in range(2):
        p.solve_f64(bd, x, k)
        S.sync_status()
        assert np.abs(x.cpu().numpy() - ref).max() <= 1e-13 * top
        x.fill_(float("nan"))
        p.solve_ir(bd, x, k)
        S.sync_status()
        assert np.abs(x.cpu().numpy() - ref).max() <= 1e-12 * top
    p.close()
    S.free_device_analysis(None, info)
