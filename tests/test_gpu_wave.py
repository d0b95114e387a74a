"""WAVE solves of stencils: lines shorter and longer than a chunk, ragged ends,
couplings into the same line, the forms that keep one row a lane, every CTA
size, block systems (in place as well), updated values and infinities."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _stencil(nx, ny, offs, seed=0, far=None):
    """Rows of an nx x ny grid that read (dx, dy) of offs, then their diagonal (dominant)."""
    rng = np.random.default_rng(seed)
    rows = []
    for j in range(ny):
        for i in range(nx):
            r = [(j + b) * nx + i + a for a, b in offs if 0 <= i + a < nx and 0 <= j + b]
            if far and i >= far:
                r.append(j * nx + i - far)
            rows.append(sorted(r) + [j * nx + i])
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    ci = np.concatenate(rows).astype(np.int32)
    va = rng.uniform(-1, 1, ci.size)
    last = rp[1:] - 1
    va[last] = 0
    va[last] = 1 + np.add.reduceat(np.abs(va), rp[:-1])
    return gen.from_arrays(rp, ci, va)


FIVE, NINE = [(-1, 0), (0, -1)], [(-1, 0), (-1, -1), (0, -1), (1, -1)]
MATS = {
    **{f"grid_{nx}": (lambda nx=nx: gen.grid2d(nx, 61, seed=1)) for nx in (2, 3, 31, 32, 127, 128, 129, 300)},
    "grid3d": lambda: gen.grid3d(37, 12, 13, seed=3),
    "four_couplings": lambda: _stencil(150, 40, NINE + [(0, -2)], seed=2),
    "nine_points": lambda: _stencil(67, 33, NINE, seed=3),
    "no_line_above": lambda: _stencil(90, 20, [(-1, 0)], seed=4),
    "five_couplings": lambda: _stencil(70, 30, NINE + [(0, -2), (0, -3)], seed=5),
    "far_130": lambda: _stencil(300, 30, [(-1, 0)], seed=10, far=130),
    "far_40": lambda: _stencil(140, 30, FIVE, seed=6, far=40),
    "far_100": lambda: _stencil(140, 30, FIVE, seed=7, far=100),
}


def _plan(S, torch, m):
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (m.rowptr, m.colidx, m.val)]
    L = S.SpMat(m.n, m.n, m.nnz, *(a.data_ptr() for a in t))
    info = S.AnalysisInfo()
    info.mode = S.ORDER
    S.run_analysis(info, L)
    return S.Plan(L, info), info, L, t


@pytest.mark.parametrize("name", list(MATS))
def test_wave_matches_the_oracle(torch_cuda, name):
    torch = torch_cuda
    import sptrsv_b200 as S

    m = MATS[name]()
    b = m.matvec(gen.vector(m.n, "uniform", seed=11))
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    top = np.abs(ref).max()
    p, info, L, keep = _plan(S, torch, m)
    bd = torch.from_numpy(b).cuda()
    x = torch.empty_like(bd)
    x32 = torch.empty(m.n, dtype=torch.float32, device="cuda")
    hb, hx = torch.from_numpy(b).pin_memory(), torch.zeros(m.n, dtype=torch.float64).pin_memory()

    def off(v):
        S.sync_status()
        return float(np.abs(v.cpu().numpy() - ref).max() / top)

    for G in (2, 4, 8, 16):
        for parts in (0, 2, 5):
            try:
                p.set_schedule(variant=S._lib.VAR_WAVE, block_warps=G, partitions=parts, ir_max_iters=2)
            except S._lib.SptrsvError as e:
                assert parts and e.code == -9 and name not in ("grid_300", "nine_points"), (G, parts, e)
                continue
            for v in (x, x32):
                v.fill_(float("nan"))
            p.solve_f64(bd, x)
            assert off(x) <= 1e-12, (G, parts)
            p.solve_ir(bd, x)
            assert off(x) <= 1e-12, (G, parts)
            p.solve_f32(bd, x32)
            assert off(x32) <= 1e-4, (G, parts)
            hx.fill_(float("nan"))
            p.solve_host(hb, hx, 1, precision=64)
            assert off(hx) <= 1e-12, (G, parts)
            if parts and p.partition_info()["blocks"] > 1:
                x.copy_(bd)
                p.solve_f64(x, x)
                assert off(x) <= 1e-12, (G, parts)
    p.close()
    S.free_device_analysis(None, info)


def test_wave_values_update(torch_cuda):
    """Block systems take updated values."""
    torch = torch_cuda
    import sptrsv_b200 as S

    calm = _stencil(300, 30, FIVE, seed=8)
    x = torch.empty(calm.n, dtype=torch.float64, device="cuda")
    p, info, L, keep = _plan(S, torch, calm)
    p.set_schedule(variant=S._lib.VAR_WAVE, block_warps=4, partitions=2)
    first = calm.val.copy()
    xt = gen.vector(calm.n, "uniform", seed=5)
    for val in (first, np.where(first < 0, 0.5 * first, first), 2 * first, first):
        calm.val[:] = val
        b = calm.matvec(xt)
        ref = O.solve(calm.rowptr, calm.colidx, calm.val, b)
        keep[2].copy_(torch.from_numpy(calm.val).cuda())
        p.update_values(L)
        p.solve_f64(torch.from_numpy(b).cuda(), x)
        S.sync_status()
        assert np.abs(x.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
    p.close()
    S.free_device_analysis(None, info)


@pytest.mark.parametrize("parts", [0, 2])
def test_wave_infinities(torch_cuda, parts):
    """An infinite b: the rest of its line as in a solve row by row (products over a few
    dozen rows underflow), every other line untouched."""
    torch = torch_cuda
    import sptrsv_b200 as S

    m = _stencil(300, 20, [(-1, 0)], seed=9)
    off = np.ones(m.nnz, bool)
    off[m.rowptr[1:] - 1] = False
    m.val[off] = 1e-9
    b = m.matvec(gen.vector(m.n, "uniform", seed=1))
    b[[905, 4390]] = np.inf, -np.inf
    ref = O.solve(m.rowptr, m.colidx, m.val, b)
    assert np.isinf(ref).sum() > 300
    p, info, L, keep = _plan(S, torch, m)
    p.set_schedule(variant=S._lib.VAR_WAVE, block_warps=4, partitions=parts)
    x = torch.empty(m.n, dtype=torch.float64, device="cuda")
    p.solve_f64(torch.from_numpy(b).cuda(), x)
    S.sync_status()
    got = x.cpu().numpy()
    fin = np.isfinite(ref)
    if parts:
        assert np.array_equal(got[~fin], ref[~fin])
    assert not np.isfinite(got[~fin]).any()
    assert np.abs(got[fin] - ref[fin]).max() <= 1e-12 * np.abs(ref[fin]).max()
    p.close()
    S.free_device_analysis(None, info)
