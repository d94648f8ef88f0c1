"""Passes and expansions on warp-owned tiles: the smallest grids that take them
(three tiles per SM) and one column less, tile counts that leave the ring of
buffers in every position, all fields, both directions, 1x, 2x and 4x, pairs."""
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


def _names(ctx, call):
    ctx.kernel_timing(True)
    call()
    torch.cuda.synchronize()
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    return names


@pytest.mark.parametrize("field", sorted(NTT))
@pytest.mark.parametrize("log_n,tiles", [(15, 444), (15, 440), (16, 448), (17, 592), (18, 640), (20, 512), (22, 512)])
def test_passes(ctx, field, log_n, tiles):
    cls, p, fwd, inv = NTT[field]
    n, batch = 1 << log_n, tiles >> (log_n - 13)
    x = O.lcg(batch * n, log_n + tiles, p, monty=field != "m31")
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    b = cls(ctx)
    stream = torch.cuda.current_stream().cuda_stream
    names = _names(ctx, lambda: b.forward_dev(d.data_ptr(), log_n, batch, stream))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    by_cluster = field == "m31" and log_n == 15  # short M31 columns: one cluster launch
    assert any("warp" in k for k in names) == (tiles >= 3 * sms and not by_cluster), names
    got = d.cpu().numpy().view(np.uint32)
    cols = sorted({0, batch // 2, batch - 1})
    for c in cols:
        assert np.array_equal(got[c * n:(c + 1) * n], fwd(x[c * n:(c + 1) * n])), c
    b.inverse_dev(d.data_ptr(), log_n, batch, stream)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), x)
    assert ctx.check_device_error() == 0


@pytest.mark.parametrize("log_n,batch,added", [(14, 222, 0), (14, 223, 1), (14, 224, 2), (14, 300, 3), (15, 111, 1),
                                               (16, 57, 2), (18, 14, 1), (20, 4, 1)])
@pytest.mark.parametrize("circle", [False, True])
def test_expansion(ctx, log_n, batch, added, circle):
    x = O.lcg(batch << log_n, 41 + log_n, O.M31_P)
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.empty(batch << (log_n + added), dtype=torch.int32, device="cuda")
    lde = sfntt.CircleLde(ctx) if circle else sfntt.M31Lde(ctx)
    lde.execute_dev(d.data_ptr(), out.data_ptr(), log_n, batch, added, torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy().view(np.uint32).reshape(batch, -1)
    ref = O.circle_lde if circle else O.m31_lde
    for c in sorted({0, 1, batch // 2, batch - 1}):
        assert np.array_equal(got[c], ref(x.reshape(batch, -1)[c], log_n, 1, added)), c
    assert ctx.check_device_error() == 0


@pytest.mark.parametrize("log_n,batch", [(14, 111), (16, 29), (18, 8)])
def test_pairs(ctx, log_n, batch):
    x = O.lcg(2 * batch << log_n, 43, O.M31_P)
    d = torch.from_numpy(x.view(np.int32).copy()).cuda()
    e = sfntt.Cm31Ntt(ctx)
    stream = torch.cuda.current_stream().cuda_stream
    e.forward_dev(d.data_ptr(), log_n, batch, stream)
    got, n2 = d.cpu().numpy().view(np.uint32), 2 << log_n
    for c in (0, batch - 1):
        assert np.array_equal(got[c * n2:(c + 1) * n2], O.cm31_ntt(x[c * n2:(c + 1) * n2], log_n, 1)), c
    e.inverse_dev(d.data_ptr(), log_n, batch, stream)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), x)
