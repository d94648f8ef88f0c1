"""One-launch LDE of short columns: every size of its range, batches around
whole tiles and around the points where output blocks get their own CTAs, every
blow-up, in-place columns (the natural-order route), and the sizes either side."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

SIZES = [(4, 7, 1)] + [(log_n, b, added) for log_n in range(5, 15) for b, added in ((1, 1), (3, 0), (5, 4), (67, 2))]
SIZES += [(5, 4099, 1), (8, 1201, 1), (9, 601, 3), (11, 593, 1), (12, 299, 1), (13, 149, 1), (14, 74, 1), (14, 75, 1)]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


def _run(lde, x, log_n, batch, added, **kw):
    d_in = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.full(((batch << (log_n + added)) + 16,), 99, dtype=torch.int32, device="cuda")
    lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, batch, added, **kw,
                    stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert (out[-16:] == 99).all()
    assert np.array_equal(d_in.cpu().numpy().view(np.uint32), x)
    return out[:-16].cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("log_n,batch,added", SIZES)
@pytest.mark.parametrize("field", ["bb", "kb"])
def test_monty(ctx, field, log_n, batch, added):
    p = O.KB_P if field == "kb" else O.BB_P
    shift = 12345 if added == 2 else 0
    x = O.lcg(batch << log_n, 17 + log_n, p, monty=True)
    lde = (sfntt.KbCosetLdeBatch if field == "kb" else sfntt.CosetLdeBatch)(ctx)
    ref = (O.kb_coset_lde if field == "kb" else O.bb_coset_lde)(x, log_n, batch, added, shift_monty=shift, threads=8)
    assert np.array_equal(_run(lde, x, log_n, batch, added, shift_monty=shift), ref)


@pytest.mark.parametrize("log_n,batch,added", SIZES)
def test_m31(ctx, log_n, batch, added):
    x = O.lcg(batch << log_n, 23 + log_n, O.M31_P)
    ref = O.m31_lde(x, log_n, batch, added, threads=8)
    assert np.array_equal(_run(sfntt.M31Lde(ctx), x, log_n, batch, added), ref)


@pytest.mark.parametrize("log_n,batch,added", [(6, 33, 2), (9, 2, 3), (12, 5, 2), (13, 3, 2), (14, 3, 2)])
def test_natural_order_in_place(ctx, log_n, batch, added):
    def rev(k):
        i = np.arange(1 << k)
        r = np.zeros_like(i)
        for b in range(k):
            r = (r << 1) | ((i >> b) & 1)
        return r
    x = O.lcg(batch << log_n, 29, O.BB_P, monty=True)
    br = x.reshape(batch, -1)[:, rev(log_n)].reshape(-1).copy()
    ref = O.bb_coset_lde(br, log_n, batch, added, threads=8).reshape(batch, -1)[:, rev(log_n + added)].reshape(-1)
    assert np.array_equal(_run(sfntt.CosetLdeBatch(ctx, natural=True), x, log_n, batch, added), ref)


@pytest.mark.parametrize("log_n", [12, 13, 14])
def test_capture_after_a_call_with_another_batch(log_n):
    """Tables resident from an ordinary call serve a capture of any batch."""
    c = sfntt.Context(0)
    lde = sfntt.CosetLdeBatch(c)
    big, few = 300, 4
    x = O.lcg(big << log_n, 31, O.BB_P, monty=True)
    ref = O.bb_coset_lde(x[:few << log_n], log_n, few, 1, threads=8)
    d_in = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.empty(big << (log_n + 1), dtype=torch.int32, device="cuda")
    lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, big, 1, stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    out.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, few, 1, stream=torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out[:few << (log_n + 1)].cpu().numpy().view(np.uint32), ref)
    del g
    c.close()
