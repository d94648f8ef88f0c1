"""LDEs whose input lies in the output buffer: the one-launch form of short columns
leaves them to the passes (checked on the host, no GPU), and their results are the
oracle's."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_one_launch_form_refuses_overlapping_buffers(tmp_path):
    lib = ROOT / "small-field-metal-ntt_b200" / "lib"
    exe = tmp_path / "test_overlap"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-I/usr/local/cuda/include", str(ROOT / "tests" / "cpp" / "test_overlap.cpp"),
                        "-o", str(exe), f"-L{lib}", "-lsfntt", f"-Wl,-rpath,{lib}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "all ok", r.stdout[-4000:]


@pytest.mark.gpu
@pytest.mark.parametrize("log_n", range(5, 15))
@pytest.mark.parametrize("added", [1, 2])
@pytest.mark.parametrize("field", ["bb", "kb", "m31"])
def test_input_at_the_end_of_the_output(field, log_n, added):
    """One column, extended from the last block of its own output column."""
    import sfntt
    from oracle import oracle as O
    torch = pytest.importorskip("torch")
    cls, p, ref = {"bb": (sfntt.CosetLdeBatch, O.BB_P, O.bb_coset_lde), "kb": (sfntt.KbCosetLdeBatch, O.KB_P, O.kb_coset_lde),
                   "m31": (sfntt.M31Lde, O.M31_P, O.m31_lde)}[field]
    n, n_ext = 1 << log_n, 1 << (log_n + added)
    x = O.lcg(n, 61 + log_n, p, monty=field != "m31")
    out = torch.full((n_ext + 16,), 99, dtype=torch.int32, device="cuda")
    out[n_ext - n:n_ext] = torch.from_numpy(x.view(np.int32)).cuda()
    lde = cls(sfntt.default_context(0))
    lde.execute_dev(out.data_ptr() + 4 * (n_ext - n), out.data_ptr(), log_n, 1, added,
                    stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert (out[n_ext:] == 99).all()
    assert np.array_equal(out[:n_ext].cpu().numpy().view(np.uint32), ref(x, log_n, 1, added))
