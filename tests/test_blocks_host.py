"""The analysis' device allocations, counted on the host: at no range of sizes
does an analysis make the driver open more chunks than it would with every array
by itself."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

DRIVER = r"""
#include <cstdio>
#include <vector>
#include "blocks.h"
using namespace sptrsv;
// the driver as measured: blocks of up to 1 MB into 2-MB chunks, first fit, larger ones alone; `room` bytes are left in a chunk that is there
struct Driver {
    std::vector<long long> left;
    int opened = 0;
    explicit Driver(long long room) : left{room} {}
    void take(long long bytes)
    {
        if (bytes <= 1 << 20) {
            for (long long& l : left)
                if (l >= bytes) { l -= bytes; return; }
            left.push_back((2 << 20) - bytes);
        }
        opened++;
    }
};
int main()
{
    int all = 0, more = 0, fewer = 0, most = 0;
    for (long long room = 0; room <= 2000000; room += 250000)
        for (long long n = 1000; n < 3000000; n += 499 + n / 500)
            for (long long warps : {n / 32 + 1, n / 4 + 1, n / 2 + 1}) {
                const long long scr = (n / 4096 + 1) * 16 + 64, lev = 32;
                const std::vector<std::vector<long long>> groups = {
                    {n + 64, n, n}, {n, n, n, scr + 64}, {7 * lev + 1, lev + 1, lev + 1, 64}, {warps, warps, warps}};
                Driver apart(room), here(room);
                for (int i = 0; i < 4; i++) {
                    const auto& g = groups[i];
                    long long sum = 0;
                    for (long long k : g) {
                        apart.take(4 * block_part(k));
                        sum += 4 * block_part(k);
                    }
                    if (share_block(g.data(), (int)g.size(), i < 2 ? kRowShare : kOtherShare)) here.take(sum);
                    else
                        for (long long k : g) here.take(4 * block_part(k));
                }
                const int d = here.opened - apart.opened;
                all++;
                more += d > 0;
                fewer += d < 0;
                if (d > most) most = d;
            }
    printf("%d %d %d %d\n", all, more, fewer, most);
    return 0;
}
"""


def test_sharing_opens_no_more_chunks_than_arrays_apart(tmp_path):
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{ROOT / 'sptrsv_b200' / 'csrc'}", str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True)
    total, more, fewer, most = map(int, r.stdout.split())
    assert most <= 1 and more <= total / 200  # now and then an array would have slipped into a gap
    assert fewer >= total / 3
