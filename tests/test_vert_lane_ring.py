"""The per-lane row rings of the vertical cross-aggregation kernels (k_vert_dual, k_cross_vol),
checked on the CPU: tests/native/vert_lane_ring_check.cpp includes the kernel's own
header (rtstereo_gb300/csrc/rts_vert_ring.h) and replays ticks, slots and walks."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_vert_lane_ring(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    exe = str(tmp_path / "vert_lane_ring_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "rtstereo_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "vert_lane_ring_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("ok")
