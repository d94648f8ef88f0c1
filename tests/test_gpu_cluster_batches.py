"""Cluster transforms at the edges of their rule: one column, a few, the last
batch that takes the clusters and the first that does not, every field."""
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


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("field", sorted(NTT))
@pytest.mark.parametrize("log_n", [13, 14, 15, 16])
@pytest.mark.parametrize("which", ["one", "five", "last", "beyond"])
def test_batches(ctx, field, log_n, which):
    cls, p, fwd, inv = NTT[field]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = (4 if log_n == 16 else 16 if field == "m31" else 3) * sms >> (log_n - 12)
    batch = {"one": 1, "five": 5, "last": last, "beyond": last + 1}[which]
    n = 1 << log_n
    x = O.lcg(batch * n, log_n + batch, p, monty=field != "m31")
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    b = cls(ctx)
    stream = torch.cuda.current_stream().cuda_stream
    ctx.kernel_timing(True)
    b.forward_dev(d.data_ptr(), log_n, batch, stream)
    torch.cuda.synchronize()
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    assert any("cluster" in k for k in names) == (which != "beyond"), names
    got = d.cpu().numpy().view(np.uint32)
    for c in sorted({0, batch // 2, batch - 1}):
        assert np.array_equal(got[c * n:(c + 1) * n], fwd(x[c * n:(c + 1) * n])), c
    b.inverse_dev(d.data_ptr(), log_n, batch, stream)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), x)
    d.copy_(torch.from_numpy(x.view(np.int32)))
    b.inverse_dev(d.data_ptr(), log_n, batch, stream)
    got = d.cpu().numpy().view(np.uint32)
    for c in sorted({0, batch - 1}):
        assert np.array_equal(got[c * n:(c + 1) * n], inv(x[c * n:(c + 1) * n])), c
