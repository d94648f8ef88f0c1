"""The rule for launching a strided pass before the previous kernel ends: passes of
up to four layers only as grids of one round (host check of csrc/pdl.cuh)."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_short_strided_passes(tmp_path):
    exe = tmp_path / "test_early_launch"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-I/usr/local/cuda/include",
                        str(ROOT / "tests" / "cpp" / "test_early_launch.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "all ok", r.stdout
