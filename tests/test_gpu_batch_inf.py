"""Infinities and NaN in the sequential systems of a batch: a row takes them from
the rows it reads and from no other."""
import numpy as np
import pytest

from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _matrix(n, per_row, seed):
    """Rows of up to per_row columns, 1 to 60 back; a fresh start every 150 rows."""
    rng = np.random.default_rng(seed)
    rows = [sorted({i - d for d in rng.choice([1, 2, 3, 4, 5, 6, 7, 9, 20, 40, 60], per_row) if i - d >= i - i % 150})
            for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(r + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = rng.uniform(0.1, 0.2, ci.size)
    va[rp[1:] - 1] = 1.0
    return gen.from_arrays(rp, ci, va)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("block_warps", [8, 4, 2])
def test_infinities_spread_as_in_substitution(torch_cuda, block_warps, precision):
    torch = torch_cuda
    import sptrsv_b200 as S
    from sptrsv_b200.batch import Batch

    ks = [1, 3, 2, 9]
    ms = [_matrix(900 + 37 * j, per, seed=j) for j, per in enumerate((1, 1, 2, 3))]
    refs, bs = [], []
    for m, k in zip(ms, ks):
        b = np.ones((m.n, k))
        b[152:160, 0], b[302:312, -1], b[455:458, 0] = np.inf, -np.inf, np.nan
        x = b.copy()
        with np.errstate(invalid="ignore"):
            for i in range(m.n):
                for p in range(m.rowptr[i], m.rowptr[i + 1] - 1):
                    x[i] -= m.val[p] * x[m.colidx[p]]
        bs.append(b.ravel())
        refs.append(x.ravel())
    assert np.isinf(refs[0]).sum() > 20
    dev = [S.allocate_memory(m.rowptr, m.colidx, m.val, m.n) for m in ms]
    B = Batch(dev, ks)
    B.set_seq_width(1e9)
    B.set_schedule(mode=2, block_warps=block_warps, ir_iters=0)
    b = torch.from_numpy(np.concatenate(bs)).cuda()
    x = torch.zeros_like(b)
    B.solve(b, x, precision)
    S.sync_status()
    got, ref = x.cpu().numpy(), np.concatenate(refs)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(got), got, 0), np.where(np.isinf(ref), ref, 0))
    fin = np.isfinite(ref)
    assert np.allclose(got[fin], ref[fin], rtol=1e-11 if precision == 64 else 1e-3, atol=1e-11 if precision == 64 else 1e-4)
    B.close()
    for d in dev:
        S.free_device_analysis(d, None)
