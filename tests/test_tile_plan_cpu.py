"""The tile partition of the implicit sweeps, checked on the host with the
kernel's own address arithmetic (tests/tiles/plan_check.cpp): slots, halo
lines, edge records, waves of zeros and ticket order, for both precisions."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = [(12, 12, 12), (97, 49, 33), (12, 13, 129), (13, 12, 130), (12, 131, 12), (136, 80, 43), (65, 129, 129),
         (33, 70, 25), (16, 16, 200), (31, 32, 12), (260, 40, 12), (129, 33, 17)]


def test_tile_plans(tmp_path):
    exe = str(tmp_path / "plan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "orion_b200", "csrc"),
                    os.path.join(ROOT, "tests", "tiles", "plan_check.cpp"), "-o", exe], check=True)
    for s in SIZES:
        r = subprocess.run([exe, *map(str, s)], capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
