"""The kernels whose warps wait on their own (warp-owned tiles, two columns at
once), one CTA on host threads: the kernel headers are compiled with g++ beside
stand-ins for the PTX ones (tests/cpp/cta), and a bulk copy or an arrival that
never lands has to end the CTA after one wait per thread, with the error flag set
and no output written after it."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "small-field-metal-ntt_b200" / "csrc"


def test_a_lost_copy_or_arrival_ends_the_cta(tmp_path):
    src = tmp_path / "pkg" / "csrc"
    src.mkdir(parents=True)
    (tmp_path / "include").mkdir()
    shutil.copy(ROOT / "include" / "sfntt.h", tmp_path / "include")
    for name in ("field.cuh", "ntt_pass.cuh", "tile_tma.cuh", "tile_warp.cuh"):
        shutil.copy(CSRC / name, src)
    for f in (ROOT / "tests" / "cpp" / "cta").iterdir():  # pdl.cuh and tma.cuh among them
        shutil.copy(f, src)
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-I/usr/local/cuda/include", "test_bounded.cpp",
                        "-o", "test_bounded"], cwd=src, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(src / "test_bounded")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "all ok", r.stdout[-4000:]
