"""Levels by 256-row groups, one thread per row: sizes around the warp and the
group, rows longer than a poll round inside and outside their warp, grid lines
that start inside a warp, and a batch whose tasks start at any row."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu


def _from_rows(rows):
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(sorted(r) + [i], dtype=np.int32) for i, r in enumerate(rows)])
    va = np.where(ci == np.repeat(np.arange(len(rows)), np.diff(rp)), 4.0, -0.01)
    return gen.from_arrays(rp, ci, va)


def _arrow(n):
    """Every 40th row reads all rows of its warp and 200 before it; the others the row before or none."""
    return _from_rows([list(range(max(0, i - 230), i)) if i % 40 == 39 else ([i - 1] if i % 3 else []) for i in range(n)])


def _nine_point(nx, ny):
    rows = []
    for j in range(ny):
        for i in range(nx):
            r = [(j - 1) * nx + i + d for d in (-1, 0, 1) if j and 0 <= i + d < nx]
            rows.append(r + ([j * nx + i - 1] if i else []))
    return _from_rows(rows)


MATS = {
    **{f"chain_{n}": (lambda n=n: _from_rows([[i - 1] if i else [] for i in range(n)])) for n in (31, 32, 33, 256, 257)},
    **{f"grid_{nx}": (lambda nx=nx: gen.grid2d(nx, 70, seed=1)) for nx in (5, 31, 32, 33, 255, 257)},
    "nine_point": lambda: _nine_point(45, 41),
    "nine_point_short": lambda: _nine_point(7, 90),
    "grid3d_short": lambda: gen.grid3d(9, 11, 13, seed=3),
    "dense_band": lambda: gen.banded(1500, 20, 20, 20, seed=5),
    "wide_band": lambda: gen.banded(3001, 900, 0, 24, seed=6),
    "block_48": lambda: gen.blockdiag(1000, 48, seed=4),
    "arrow": lambda: _arrow(777),
}


@pytest.mark.parametrize("name", list(MATS))
def test_levels_match_the_oracle(torch_cuda, name):
    import sptrsv_b200 as S

    m = MATS[name]()
    ref = O.analysis(m.rowptr, m.colidx)
    L = S.allocate_memory(m.rowptr, m.colidx, m.val, m.n)
    info = S.AnalysisInfo()
    info.mode = S.MULTIROW
    assert S.run_analysis(info, L) == 0
    got = S.analysis_arrays(info, m.n)
    S.free_device_analysis(L, info)
    assert got["nlevs"] == ref["nlevs"]
    for k in ("levels", "iorder", "ibase_row", "ivect_size_warp"):
        assert np.array_equal(got[k], ref[k]), k


def test_batch_union_of_unaligned_systems(torch_cuda):
    import sptrsv_b200 as S
    from sptrsv_b200.batch import Batch

    sizes = [1, 31, 255, 256, 257, 700, 1025]
    ms = [gen.banded(n, 40, 2, 12, seed=n) for n in sizes]
    mats = [S.allocate_memory(m.rowptr, m.colidx, m.val, m.n) for m in ms]
    B = Batch(mats, [1] * len(ms))
    assert B.nlevs == max(O.analysis(m.rowptr, m.colidx)["nlevs"] for m in ms)
    for L in mats:
        S.free_device_analysis(L, None)
