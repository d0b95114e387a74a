"""BAND's steps: rows of every length in one unit, a unit whose list schedule
keeps more values alive than there are slots (its steps then follow the
levels), units of fewer steps than warps, and solves in place."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _from_rows(rows, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(sorted(r) + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = rng.uniform(-1, 1, ci.size)
    last = rp[1:] - 1
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1])
    return gen.from_arrays(rp, ci, va)


def _chains_with_leaves(chains, length):
    """Chains side by side; every chain row is also read by a leaf, which the chains' rows come before."""
    rows = []
    for k in range(length):
        top = 2 * chains * k
        rows += [[top + c - 2 * chains] if k else [] for c in range(chains)]
        rows += [[top + c] for c in range(chains)]
    return _from_rows(rows, 3)


MATS = {
    "all_lengths": lambda: gen.banded(6000, 200, 0, 128, seed=3),
    "few_steps": lambda: gen.banded(300, 40, 0, 3, seed=4),
    "one_row": lambda: gen.from_arrays([0, 1], [0], [3.0]),
    "slots_run_out": lambda: _chains_with_leaves(40, 260),
}


@pytest.mark.parametrize("name", list(MATS))
def test_band_steps_match_the_oracle(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = MATS[name]()
    b = m.matvec(gen.vector(m.n, "uniform", seed=5))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ALL
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(variant=S._lib.VAR_BAND, ir_max_iters=2)
    bd = torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    for solve in (p.solve_f64, p.solve_ir):
        x.fill_(float("nan"))
        solve(bd, x)
        S.sync_status()
        assert O.rel_err(x.cpu().numpy(), ref) <= 1e-12
    p.close()
    S.free_device_analysis(L, info)


@pytest.mark.parametrize("P", [0, 24])
def test_band_solves_in_place(torch_cuda, P):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = gen.banded(30000, 256, 8, 8, seed=0)
    b = m.matvec(gen.vector(m.n, "uniform", seed=6))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ALL
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(variant=S._lib.VAR_BAND, partitions=P)
    for _ in range(2):
        x = torch.from_numpy(b).cuda()
        p.solve_f64(x, x)
        S.sync_status()
        assert O.rel_err(x.cpu().numpy(), ref) <= 1e-12
    p.close()
    S.free_device_analysis(L, info)
