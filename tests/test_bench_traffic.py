"""The DRAM traffic that bench.py prints beside a roofline: only of a capture of
the kernel and schedule that ran, and every capture names a kernel of the library;
and which matrices it counts one launch a partitioned WAVE solve for."""
import json
import re
from pathlib import Path

import bench
from sptrsv_b200 import gen

ROOT = Path(__file__).resolve().parent.parent


def test_traffic_is_of_the_schedule_that_ran():
    caught = json.loads((ROOT / "profiles" / "ncu_traffic.json").read_text())
    sources = "".join(p.read_text() for p in (ROOT / "sptrsv_b200" / "csrc").iterdir() if p.is_file())
    for key, entry in caught.items():
        for schedule in entry["schedules"]:
            assert bench.load_traffic(key, schedule) == entry["dram_bytes_per_launch"]
        assert bench.load_traffic(key, "another") is None
        name = re.match(r"\w+", entry["kernel"]).group()
        assert re.search(rf"\b{name}\(", sources), name
        for doc in re.findall(r"profiles/\S+\.md", entry["source"]):
            text = (ROOT / doc).read_text()
            assert text.splitlines()[0].startswith(f"# {name}")
            assert "Taken with an earlier form" not in text
    assert bench.load_traffic("no_such_key", "wave/G4-P16") is None
    # the kernel that a partitioned WAVE solve of the grid launches
    assert caught["wave_p16_f64_c1"]["kernel"].startswith("k_sptrsv_wave4<")


def test_one_coupling():
    assert bench.one_coupling(gen.grid2d(13, 9, seed=1))
    assert not bench.one_coupling(gen.grid3d(5, 4, 3, seed=1))
    assert not bench.one_coupling(gen.banded(200, 16, 4, 8, seed=1))
