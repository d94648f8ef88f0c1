"""Barrier ids of the tile engine's exchanges where a kernel runs the inverse and
then the forward layers of a tile (short-column LDE, natural-order expansion): an
id must stand for the same threads in both.  The kernel headers are compiled with
g++ beside stand-ins for the PTX ones (tests/cpp/cta)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "small-field-metal-ntt_b200" / "csrc"


def test_an_id_stands_for_one_set_of_threads(tmp_path):
    src = tmp_path / "pkg" / "csrc"
    src.mkdir(parents=True)
    (tmp_path / "include").mkdir()
    shutil.copy(ROOT / "include" / "sfntt.h", tmp_path / "include")
    for name in ("field.cuh", "ntt_pass.cuh", "tile_tma.cuh"):
        shutil.copy(CSRC / name, src)
    for name in ("cta.hpp", "pdl.cuh", "tma.cuh", "test_barriers.cpp"):
        shutil.copy(ROOT / "tests" / "cpp" / "cta" / name, src)
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-I/usr/local/cuda/include", "test_barriers.cpp",
                        "-o", "test_barriers"], cwd=src, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(src / "test_barriers")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "all ok", r.stdout[-4000:]
