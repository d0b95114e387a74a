"""The BAND schedule's steps and slots, built on the host: rows come after the
rows they read, steps and slots hold what they may, and narrow matrices are cut
in time linear in their entries."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from sptrsv_b200 import gen

ROOT = Path(__file__).resolve().parent.parent

DRIVER = r"""
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include "band_steps.h"
using namespace sptrsv;
// argv: n, row pointers, columns, levels (int32 files); prints seconds, steps and the cheaper level cut's steps
static std::vector<int> read(const char* path)
{
    FILE* f = fopen(path, "rb");
    fseek(f, 0, SEEK_END);
    std::vector<int> v(ftell(f) / 4);
    rewind(f);
    if (fread(v.data(), 4, v.size(), f) != v.size()) exit(9);
    fclose(f);
    return v;
}
int main(int, char** argv)
{
    const int n = atoi(argv[1]);
    std::vector<int> rp = read(argv[2]), ci = read(argv[3]), lev = read(argv[4]);
    BandUnit u, l;
    auto t = std::chrono::steady_clock::now();
    band_unit(rp.data(), ci.data(), lev.data(), 0, n, u);
    const double sec = std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
    band_level_steps(rp.data(), lev.data(), 0, n, l);
    // a row's columns in earlier steps, lanes enough, every row once
    std::vector<int> step(n, -1), holds(u.R, -1);
    for (size_t k = 0; k < u.steps.size(); k++) {
        const BandStepHost& s = u.steps[k];
        if (s.cnt < 1 || s.cnt * s.kp > 32) return 1;
        for (int q = s.first; q < s.first + s.cnt; q++) {
            const int r = u.order[q], len = rp[r + 1] - 1 - rp[r];
            if (step[r] >= 0 || len > kBandU * s.kp) return 2;
            for (int e = rp[r]; e < rp[r + 1] - 1; e++) {
                if (step[ci[e]] < 0) return 3;
                if (holds[u.slot_of[ci[e]]] != ci[e]) return 4;  // its slot still holds it
            }
        }
        for (int q = s.first; q < s.first + s.cnt; q++) {
            const int r = u.order[q];
            step[r] = (int)k;
            if (u.slot_of[r] < 0 || u.slot_of[r] >= u.R) return 5;
            holds[u.slot_of[r]] = r;
        }
    }
    for (int r = 0; r < n; r++)
        if (step[r] < 0) return 6;
    printf("%f %zu %zu %d\n", sec, u.steps.size(), l.steps.size(), u.R);
    return 0;
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("band")
    (d / "t.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'sptrsv_b200' / 'csrc'}", str(d / "t.cpp"), "-o", str(d / "t")],
                   check=True)

    def run(m, timeout):
        lev = np.zeros(m.n, np.int32)
        rp, ci = m.rowptr.tolist(), m.colidx.tolist()
        level = [0] * m.n
        for i in range(m.n):
            s, e = rp[i], rp[i + 1] - 1
            level[i] = 1 + (max(level[c] for c in ci[s:e]) if e > s else 0)
        lev[:] = level
        for name, a in (("rp", m.rowptr), ("ci", m.colidx), ("lev", lev)):
            np.ascontiguousarray(a, dtype=np.int32).tofile(d / name)
        r = subprocess.run([str(d / "t"), str(m.n), *(str(d / k) for k in ("rp", "ci", "lev"))], capture_output=True,
                           text=True, timeout=timeout)
        assert r.returncode == 0, r.returncode
        sec, steps, by_level, ring = r.stdout.split()
        return float(sec), int(steps), int(by_level), int(ring)

    return run


def _rows(rows):
    rp = np.concatenate([[0], np.cumsum([len(r) + 1 for r in rows])])
    ci = np.concatenate([np.array(list(r) + [i], dtype=np.int32) for i, r in enumerate(rows)])
    return gen.from_arrays(rp, ci, np.ones(ci.size))


def _short_beside_long(n):
    """A chain, and as many rows of six entries, all ready early, which its steps have no lanes for."""
    head = [[] for _ in range(8)] + [[0, 1, 2, 3, 4, 5] for _ in range(n)]
    chain = [[] if k == 0 else [len(head) + k - 1] for k in range(n)]
    return _rows(head + chain)


SMALL = {
    "empty_rows": lambda: _rows([[] for _ in range(100)]),
    "one": lambda: _rows([[]]),
    "band": lambda: gen.banded(3000, 64, 4, 8, seed=1),
    "wide_rows": lambda: gen.banded(2000, 200, 0, 128, seed=2),
    "grid": lambda: gen.grid2d(50, 61, seed=3),
    "mixed": lambda: _short_beside_long(2000),
}


@pytest.mark.parametrize("name", list(SMALL))
def test_steps_and_slots_are_sound(cut, name):
    _, steps, by_level, ring = cut(SMALL[name](), 60)
    assert steps <= by_level and ring <= 8192


# the matrices that took 12 to 150 seconds when a step looked at every height below the ready rows'
LONG = {
    "bidiagonal": lambda: _rows([[i - 1] if i else [] for i in range(400_000)]),
    "band_16": lambda: gen.banded(400_000, 16, 4, 8, seed=4),
    "band_64": lambda: gen.banded(400_000, 64, 4, 8, seed=5),
    "mixed": lambda: _short_beside_long(200_000),
}


@pytest.mark.parametrize("name", list(LONG))
def test_long_chains_are_cut_in_linear_time(cut, name):
    sec, steps, by_level, _ = cut(LONG[name](), 10)
    assert sec < 2.0, sec
    assert steps <= by_level
