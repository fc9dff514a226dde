"""The target of a thread in the kernels whose lanes share targets
(loquat_b200/csrc/lq_lanes.h), compiled with g++ and compared with 64-bit
arithmetic for up to 2^31 - 1 targets (tests/lane_target_check.cpp); and the
kernels take it from there."""
from __future__ import annotations

import re
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_lane_target_for_every_count(tmp_path):
    exe = tmp_path / "lane_target_check"
    cmd = [shutil.which("g++") or "g++", "-std=c++17", "-O1", "-Wall", "-Werror",
           f"-I{ROOT / 'loquat_b200' / 'csrc'}", str(ROOT / "tests" / "lane_target_check.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr


def test_drop_in_kernels_use_it():
    src = (ROOT / "loquat_b200" / "csrc" / "sph.cu").read_text()
    for name in ("k_adami", "k_shepard"):
        body = src[src.index(f" {name}(const Parameters"):]
        body = body[:body.index("\n}\n")]
        assert re.search(r"= (npb \+ )?lane_target\(", body), body[:300]
