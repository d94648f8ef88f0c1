"""Short-column LDEs whose columns are a few more than the GPU holds at once: their
output blocks are split over CTAs so that the last round is not nearly empty."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _lde(field, log_n, batch, added):
    cls, p, ref = {"bb": (sfntt.CosetLdeBatch, O.BB_P, O.bb_coset_lde), "m31": (sfntt.M31Lde, O.M31_P, O.m31_lde)}[field]
    x = O.lcg(batch << log_n, 71 + log_n, p, monty=field == "bb")
    d_in = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.full(((batch << (log_n + added)) + 16,), 99, dtype=torch.int32, device="cuda")
    lde = cls(sfntt.default_context(0))
    call = lambda s: lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, batch, added, stream=s)
    return x, d_in, out, call, lambda: ref(x, log_n, batch, added, threads=8)


@pytest.mark.parametrize("field,log_n,batch,added", [("m31", 13, 150, 4), ("m31", 13, 149, 1), ("m31", 13, 200, 3),
                                                     ("bb", 13, 149, 3), ("bb", 13, 200, 2), ("m31", 12, 150, 4),
                                                     ("m31", 12, 297, 2), ("bb", 12, 149, 4), ("bb", 11, 593, 2)])
def test_values(field, log_n, batch, added):
    x, d_in, out, call, ref = _lde(field, log_n, batch, added)
    call(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert (out[-16:] == 99).all()
    assert np.array_equal(out[:-16].cpu().numpy().view(np.uint32), ref())
    assert np.array_equal(d_in.cpu().numpy().view(np.uint32), x)


def test_one_column_more_than_the_sms():
    """149 columns of 2^13 points, 16x, one CTA per SM: not twice as long as 148."""
    times = []
    for batch in (148, 149):
        _, d_in, out, call, _ = _lde("m31", 13, batch, 4)
        st = torch.cuda.Stream()
        best = float("inf")
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record(st)
            call(st.cuda_stream)
            call(st.cuda_stream)
            e1.record(st)
            st.synchronize()
            best = min(best, e0.elapsed_time(e1))
        times.append(best)
    assert times[1] < 1.75 * times[0], times
