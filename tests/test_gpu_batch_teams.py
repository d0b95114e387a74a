"""Sequential systems of a batch: teams of seven, two and one warps; reaches
past the ring; columns cut into several units; rows and chunks longer than the
staged form takes; and batches of more units than teams, one warp a unit."""
import numpy as np
import pytest

from oracle import oracle as O
from sptrsv_b200 import gen

pytestmark = pytest.mark.gpu

# (rows, bandwidth, least and most off-diagonals, right-hand sides)
SYSTEMS = {
    "reach": [(2600, 2500, 3, 9, 2), (5000, 2047, 4, 8, 3), (3001, 1030, 4, 16, 32), (1500, 1023, 4, 16, 31)],
    "long_rows": [(700, 60, 20, 60, 5), (555, 33, 33, 33, 32), (90, 80, 70, 80, 1)],
    "small": [(1, 1, 0, 0, 7), (2, 1, 1, 1, 1), (8, 3, 1, 3, 32), (55, 7, 2, 5, 4), (57, 4, 0, 4, 17), (113, 2, 1, 2, 9)],
    "chains": [(1000, 1, 1, 1, 8), (997, 3, 2, 3, 16), (4097, 16, 4, 16, 1)],
    "many": [(60 + i % 13, 5, 1, 4, 1 + i % 2) for i in range(1500)],
}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("block_warps", [8, 4, 2])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_sequential_systems_match_the_oracle(torch_cuda, name, block_warps, precision):
    torch = torch_cuda
    import sptrsv_b200 as S
    from sptrsv_b200.batch import Batch

    ms = [gen.banded(n, bw, lo, hi, seed=7 * i + 1) for i, (n, bw, lo, hi, _) in enumerate(SYSTEMS[name])]
    ks = [s[4] for s in SYSTEMS[name]]
    bs = [m.matvec(gen.vector(m.n * k, "uniform", seed=i), k) for i, (m, k) in enumerate(zip(ms, ks))]
    dev = [S.allocate_memory(m.rowptr, m.colidx, m.val, m.n) for m in ms]
    B = Batch(dev, ks)
    B.set_seq_width(1e9)
    B.set_schedule(mode=2, block_warps=block_warps)
    assert B.seq_systems()[0] == len(ms)
    b = torch.from_numpy(np.concatenate(bs)).cuda()
    x = torch.full_like(b, float("nan"))
    B.solve(b, x, precision)
    S.sync_status()
    got = x.cpu().numpy()
    for i, (m, k) in enumerate(zip(ms, ks)):
        ref = O.solve(m.rowptr, m.colidx, m.val, bs[i], nrhs=k)
        assert O.rel_err(got[B.offsets[i]:B.offsets[i + 1]], ref) <= 1e-12, i
    B.close()
    for d in dev:
        S.free_device_analysis(d, None)
