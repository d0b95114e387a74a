"""Solves in place of partitioned plans (the result over b): refined ones without
a correction, and ones that are captured after an ordinary solve."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu

PLANS = {
    "band": (lambda: gen.banded(40000, 64, 4, 8, seed=3), dict(variant=6, block_warps=8, partitions=32)),
    "wave": (lambda: gen.grid2d(200, 300, seed=3), dict(variant=5, block_warps=4, partitions=4)),
    "wave3d": (lambda: gen.grid3d(40, 20, 300, seed=3), dict(variant=5, block_warps=4, partitions=2)),
}


@pytest.mark.parametrize("name", list(PLANS))
def test_in_place_and_captured(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    make, sched = PLANS[name]
    m = make()
    b = m.matvec(gen.vector(m.n, "uniform", seed=4))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(ir_max_iters=0, **sched)
    bd = torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    p.solve_f64(bd, x)
    p.solve_ir(bd, x)
    for solve, tol in ((p.solve_f64, 1e-12), (p.solve_ir, 1e-4)):
        for _ in range(5):
            x.copy_(bd)
            solve(x, x)
            S.sync_status()
            assert O.rel_err(x.cpu().numpy(), ref) <= tol
        stream = torch.cuda.Stream()
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            solve(x, x, stream=stream)
        x.copy_(bd)
        graph.replay()
        S.sync_status()
        assert O.rel_err(x.cpu().numpy(), ref) <= tol
    p.close()
    S.free_device_analysis(L, info)
