"""Host calls report a device-side wait that ran out: each call that copies a
result back reads the context's error flag after its last synchronisation, or it
would return success with a part of the result never written and leave the flag
to the next call.  (No wait of the library can be made to run out from outside,
so the calls' source is read.)"""
from __future__ import annotations

import re
from pathlib import Path

CAPI = Path(__file__).resolve().parents[1] / "small-field-metal-ntt_b200" / "csrc" / "capi.cu"
NO_WAITS = {"device_flag", "sfntt_pointwise_mul"}  # the flag's own read; element-wise kernels


def _functions(text: str) -> dict[str, str]:
    """Name -> body of every function that starts in column 0."""
    out = {}
    for m in re.finditer(r"^(?:int|Status|void) (\w+)\([^;{]*\) \{\n(.*?)^\}", text, re.S | re.M):
        out[m[1]] = m[2]
    return out


def test_every_call_that_copies_back_reads_the_flag():
    bodies = {k: b for k, b in _functions(CAPI.read_text()).items() if "cudaMemcpyDeviceToHost" in b}
    assert {"run_host_ntt", "run_host_lde", "sfntt_circle_ntt", "sfntt_layout", "sfntt_cm31_ntt"} <= set(bodies)
    for name, body in bodies.items():
        if name in NO_WAITS:
            continue
        sync = body.rfind("cudaStreamSynchronize(")
        assert sync >= 0, name
        assert "device_flag(ctx)" in body[sync:], f"{name} returns without reading the error flag"
