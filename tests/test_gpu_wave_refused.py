"""A partitioned WAVE plan keeps solving after a schedule that was refused: the
refusal takes the block system's layout away, and every kind of solve builds its
own again before it chooses a kernel."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["f64", "f32", "ir", "host", "update"])
def test_solves_after_a_refused_schedule(torch_cuda, first):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = gen.grid2d(2000, 80, seed=3)  # 16 lines do not fit a CTA's shared memory, 8 do
    b = m.matvec(gen.vector(m.n, "uniform", seed=4))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    p = S.Plan(L, info)
    p.set_schedule(5, block_warps=8, partitions=2, ir_max_iters=3)
    bd = torch.from_numpy(b).cuda()
    hb = torch.from_numpy(b).pin_memory()

    def solve(kind):
        dtype = torch.float32 if kind == "f32" else torch.float64
        x = torch.full((m.n,), float("nan"), dtype=dtype, device="cpu" if kind == "host" else "cuda")
        if kind == "host":
            x = x.pin_memory()
            p.solve_host(hb, x, precision=64)
        else:
            {"f64": p.solve_f64, "f32": p.solve_f32, "ir": p.solve_ir}[kind](bd, x)
            S.sync_status()
        assert O.rel_err(x.double().cpu().numpy(), ref) <= (1e-4 if kind == "f32" else 1e-12), kind

    solve("f64")
    with pytest.raises(S.SptrsvError):
        p.set_schedule(5, block_warps=16, partitions=2)
    assert p.schedule().block_warps == 8
    if first == "update":
        p.update_values(L)
    for kind in [k for k in (first,) if k != "update"] + ["f64", "f32", "ir", "host"]:
        solve(kind)
    p.close()
    S.free_device_analysis(L, info)
