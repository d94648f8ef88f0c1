"""Cluster transforms on either side of every line between their forms: blocks of
2^12 and of 2^13 words, launched early or plainly.  Calls follow one another without
a pause (early launches overlap), and the kernel names show which form ran."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

NTT = {"bb": (sfntt.BbCudaCtGsR4, O.BB_P, O.bb_forward, O.bb_inverse),
       "kb": (sfntt.KbCudaCtGsR4, O.KB_P, O.kb_forward, O.kb_inverse),
       "m31": (sfntt.CudaCtGsR4, O.M31_P, O.m31_forward, O.m31_inverse)}
# per size: batches next to 0.35, 0.76, 1, 1.4 and 2 blocks of 2^12 words per SM (148
# SMs), and to the clusters of wide blocks that run at once
BATCHES = {13: [25, 26, 46, 47, 74, 75, 103, 104, 148, 149], 14: [12, 13, 28, 29, 51, 52, 71, 74, 75, 112, 300],
           15: [6, 7, 14, 15, 25, 26, 33, 34], 16: [3, 4, 7, 8, 12, 13, 15, 16, 28, 29]}
CASES = [(f, log_n, b) for f in sorted(NTT) for log_n, bs in BATCHES.items() for b in bs]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("field,log_n,batch", CASES)
def test_calls_in_a_row(ctx, field, log_n, batch):
    cls, p, fwd, inv = NTT[field]
    n = 1 << log_n
    x = O.lcg(batch * n, 7 * log_n + batch, p, monty=field != "m31")
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    e = d.clone()
    b = cls(ctx)
    s = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for _ in range(3):  # other data between the calls: their tiles must not mix
        b.forward_dev(d.data_ptr(), log_n, batch, s)
        b.inverse_dev(e.data_ptr(), log_n, batch, s)
        b.inverse_dev(d.data_ptr(), log_n, batch, s)
        b.forward_dev(e.data_ptr(), log_n, batch, s)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), x)
    assert np.array_equal(e.cpu().numpy().view(np.uint32), x)
    ctx.kernel_timing(True)
    b.forward_dev(d.data_ptr(), log_n, batch, s)
    b.inverse_dev(e.data_ptr(), log_n, batch, s)
    torch.cuda.synchronize()
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    got_f, got_i = d.cpu().numpy().view(np.uint32), e.cpu().numpy().view(np.uint32)
    for c in sorted({0, batch // 2, batch - 1}):
        assert np.array_equal(got_f[c * n:(c + 1) * n], fwd(x[c * n:(c + 1) * n])), c
        assert np.array_equal(got_i[c * n:(c + 1) * n], inv(x[c * n:(c + 1) * n])), c
    per_sm = (batch << (log_n - 12)) / torch.cuda.get_device_properties(0).multi_processor_count
    clusters = [k for k in names if "cluster" in k]
    wide = [k for k in clusters if k.endswith("w")]
    if field != "m31":
        if log_n == 13 and per_sm > 0.63:
            assert bool(clusters) == (per_sm % 1 == 0), names
        elif per_sm <= 3:
            assert len(clusters) == 2, names
        if per_sm <= 0.76:
            assert not wide, names
        elif log_n > 13 and per_sm <= 1.6:
            assert len(wide) == (1 if log_n == 16 else 2), names  # one per SM; not the inverse of 2^16
    elif per_sm <= 3:
        assert len(clusters) == 2, names
        assert len(wide) == (2 if 1.4 < per_sm <= 1.6 else 0) or per_sm > 1.6, names


def test_first_wide_call_inside_a_capture():
    """The form is chosen without work that a capture refuses."""
    c = sfntt.Context(0)
    b = sfntt.KbCudaCtGsR4(c)
    c.prepare(b.FIELD, 15)
    n, batch = 1 << 15, 22
    x = O.lcg(batch * n, 3, O.KB_P, monty=True)
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        b.forward_dev(d.data_ptr(), 15, batch, s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(d[:n].cpu().numpy().view(np.uint32), O.kb_forward(x[:n]))
    c.close()
