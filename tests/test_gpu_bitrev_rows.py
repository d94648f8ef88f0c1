"""Bit-reversed row-major layout on either side of the lines between the register
tiles and the TMA tiles: by columns, words and whether a row is a copy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402

# log_n, columns, TMA tiles
LINES = [(16, 71, False), (16, 72, True), (15, 72, False), (16, 73, False), (16, 96, False), (17, 73, True), (17, 96, True),
         (17, 100, False), (18, 97, False), (18, 99, False), (18, 100, True), (18, 127, False), (18, 128, True),
         (19, 97, True), (15, 128, False), (15, 129, True), (15, 192, True), (14, 192, False), (15, 193, False),
         (16, 193, False), (16, 196, True), (16, 255, False), (17, 193, True), (16, 256, True), (15, 256, False)]


def _bitrev(k):
    r = np.zeros(1 << k, dtype=np.int64)
    for i in range(k):
        r |= ((np.arange(1 << k) >> i) & 1) << (k - 1 - i)
    return torch.from_numpy(r).cuda()


@pytest.mark.parametrize("log_n,batch,tma", LINES)
def test_lines(log_n, batch, tma):
    ctx = sfntt.default_context(0)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(log_n * 1000 + batch)
    n = 1 << log_n
    x = torch.randint(0, 1 << 31, (batch * n,), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    out = torch.full((batch * n + 64,), 7, dtype=torch.int32, device="cuda")
    ctx.kernel_timing(True)
    sfntt.layout_dev(ctx, x.data_ptr(), out.data_ptr(), log_n, batch, sfntt.LAYOUT_NATURAL | sfntt.LAYOUT_ROW_MAJOR,
                     torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    assert names == ["layout_transpose_bitrev" + ("_tma" if tma else "")]
    ref = x.view(batch, n).t().contiguous()[_bitrev(log_n)]  # row R holds the words at bitrev(R)
    assert torch.equal(out[:-64].view(n, batch), ref)
    assert (out[-64:] == 7).all()
    assert ctx.check_device_error() == 0
