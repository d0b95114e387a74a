"""Two host threads, each with its own matrix, stream and vectors: the shared
memory that one thread's launch takes is no limit for the other's."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _in_two_threads(torch, S, jobs, loops):
    """jobs: (solve(x, stream), reference) each; the first wrong or failed pass of each thread."""
    gate, bad = threading.Barrier(len(jobs)), [None] * len(jobs)

    def work(k):
        solve, ref = jobs[k]
        stream = torch.cuda.Stream()
        x = torch.empty(ref.size, dtype=torch.float64, device="cuda")
        gate.wait()
        for i in range(loops):
            try:
                with torch.cuda.stream(stream):
                    x.fill_(float("nan"))
                    solve(x, stream.cuda_stream)
                    got = x.cpu().numpy()
                assert O.rel_err(got, ref) <= 1e-12
            except Exception as e:
                bad[k] = (i, e)
                return

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert bad == [None] * len(jobs)


def _system(torch, S, m):
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ALL
    assert S.run_analysis(info, L) == 0
    b = m.matvec(gen.vector(m.n, "uniform", seed=5))
    return L, info, torch.from_numpy(b).cuda(), O.solve(m.rowptr, m.colidx, m.val, b)


@pytest.mark.parametrize("solver", ["order", "multirow", "lines"])
def test_drop_in_solves_from_two_threads(torch_cuda, solver):
    torch = torch_cuda
    import sptrsv_b200 as S

    ms = ([gen.grid2d(200, 200, seed=1), gen.grid2d(1500, 150, seed=2)] if solver == "lines"
          else [gen.banded(5000, 64, 4, 8, seed=1), gen.banded(20000, 64, 4, 8, seed=2)])
    call = S.csr_L_solve_multirow if solver == "multirow" else S.csr_L_solve_order
    sys_ = [_system(torch, S, m) for m in ms]
    jobs = [(lambda x, st, L=L, info=info, b=b, n=m.n: call(L, info, b, x, n, st), ref)
            for m, (L, info, b, ref) in zip(ms, sys_)]
    _in_two_threads(torch, S, jobs, 400)
    for L, info, _, _ in sys_:
        S.free_device_analysis(L, info)


PLANS = {
    "strip": [dict(variant=4, rows_per_warp=8, block_warps=16), dict(variant=4, rows_per_warp=16, block_warps=16)],
    "wave": [dict(variant=5, block_warps=8)] * 2,
    "level": [dict(variant=1, rows_per_warp=32)] * 2,
}


@pytest.mark.parametrize("name", list(PLANS))
def test_plans_from_two_threads(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    ms = [gen.grid2d(600, 16, seed=1), gen.grid2d(2000, 10, seed=2)]
    jobs, keep = [], []
    for m, sched in zip(ms, PLANS[name]):
        L, info, b, ref = _system(torch, S, m)
        p = S.Plan(L, info)
        p.set_schedule(**sched)
        keep.append((p, L, info))
        jobs.append((lambda x, st, p=p, b=b: p.solve_f64(b, x, stream=st), ref))
    _in_two_threads(torch, S, jobs, 400)
    for p, L, info in keep:
        p.close()
        S.free_device_analysis(L, info)
