"""Narrow systems solved level by level by one CTA: every lane count and team
size, x whole in shared memory and in the ring (with columns that left it),
levels wider than a team, rows longer than the loads ahead, every precision."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _with_long_rows(n, every, length):
    """A band of 3 in which every `every`-th row reads `length` rows back to the start."""
    rows = []
    for i in range(n):
        c = set(range(max(0, i - 3), i))
        if i % every == every - 1:
            c |= set(np.linspace(0, i - 1, min(i, length)).astype(int).tolist())
        rows.append(sorted(c))
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(r + [i], dtype=np.int32) for i, r in enumerate(rows)])
    rng = np.random.default_rng(n)
    va = rng.uniform(-1, 1, ci.size)
    last = rp[1:] - 1
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1])
    return gen.from_arrays(rp, ci, va)


def _wide_now_and_then(n):
    """A chain of blocks: 200 rows that read one, then one that reads 8 of them."""
    rows = []
    for i in range(n):
        j = i % 201
        rows.append([i - j - 1] if j < 200 and i > j else (list(range(i - 8, i)) if j == 200 else []))
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(r + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = np.where(ci == np.repeat(np.arange(n), np.diff(rp)), 3.0, -0.3)
    return gen.from_arrays(rp, ci, va)


MATS = {
    "one_lane": lambda: gen.banded(700, 12, 1, 3, seed=1),
    "two_lanes": lambda: gen.banded(5000, 64, 4, 8, seed=2),
    "four_lanes": lambda: gen.banded(4001, 200, 9, 16, seed=3),
    "eight_lanes": lambda: gen.banded(900, 40, 25, 32, seed=4),
    "teams_of_2": lambda: gen.banded(20000, 256, 8, 8, seed=0),
    "teams_of_4": lambda: gen.banded(24999, 1000, 8, 8, seed=5),
    "teams_of_8": lambda: gen.banded(25700, 1500, 10, 16, seed=6),
    "ring": lambda: gen.banded(40003, 300, 4, 8, seed=7),
    "ring_far_columns": lambda: _with_long_rows(40000, 97, 5),
    "long_rows": lambda: _with_long_rows(3000, 50, 120),
    "wide_levels": lambda: _wide_now_and_then(2011),
    "small_grid": lambda: gen.grid2d(61, 47, seed=1),
    "chain": lambda: gen.grid2d(1000, 1, seed=1),
    "diagonal": lambda: gen.from_arrays(np.arange(1001), np.arange(1000), np.full(1000, 3.0)),
    "one_row": lambda: gen.from_arrays([0, 1], [0], [3.0]),
}


@pytest.mark.parametrize("name", list(MATS))
def test_narrow_solves_match_the_oracle(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = MATS[name]()
    b = m.matvec(gen.vector(m.n, "uniform", seed=11))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    top = np.abs(ref).max()
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.ALL
    S.run_analysis(info, L)
    bd = torch.from_numpy(b).cuda()
    x = torch.full_like(bd, float("nan"))

    def off():
        e = float(np.abs(x.cpu().numpy() - ref).max() / top)
        x.fill_(float("nan"))
        return e

    S.csr_L_solve_multirow(L, info, bd, x, m.n)
    assert off() <= 1e-12
    S.csr_L_solve_order(L, info, bd, x, m.n)
    assert off() <= 1e-12
    p = S.Plan(L, info)
    for variant in (1, 2):
        p.set_schedule(variant, rows_per_warp=4, ir_max_iters=2)
        p.solve_f64(bd, x)
        assert off() <= 1e-12
        p.solve_ir(bd, x)
        assert off() <= 1e-12
        x32 = torch.full((m.n,), float("nan"), dtype=torch.float32, device="cuda")
        p.solve_f32(bd, x32)
        assert float(np.abs(x32.cpu().numpy() - ref).max() / top) <= 1e-4
    S.sync_status()
    p.close()
    S.free_device_analysis(L, info)
