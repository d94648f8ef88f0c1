"""Row-major layout of the shapes that take the TMA tiles (2^22 words or more,
up to 256 columns): few and many 32-row pieces per tile, column counts that are
not a multiple of 4 or 32, both row orders, and the limits of the rule."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


def _bitrev(log_n):
    i = torch.arange(1 << log_n, device="cuda")
    r = torch.zeros_like(i)
    for b in range(log_n):
        r = (r << 1) | ((i >> b) & 1)
    return r


@pytest.mark.parametrize("log_n,batch", [(21, 2), (21, 3), (20, 7), (18, 17), (17, 32), (17, 33), (16, 71), (16, 72),
                                         (16, 75), (16, 100), (15, 129), (15, 255), (14, 256), (15, 257)])
@pytest.mark.parametrize("bitrev", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_row_major(ctx, log_n, batch, bitrev, offset):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(log_n * 1000 + batch)
    words = batch << log_n
    src = torch.randint(0, 1 << 31, (words + 4,), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    dst = torch.full((words + 8,), -1, dtype=torch.int32, device="cuda")
    x = src[offset:offset + words]
    flags = sfntt.LAYOUT_ROW_MAJOR | (sfntt.LAYOUT_NATURAL if bitrev else 0)
    sfntt.layout_dev(ctx, x.data_ptr(), dst.data_ptr() + 16, log_n, batch, flags,
                     torch.cuda.current_stream().cuda_stream)
    want = x.view(batch, -1).t()
    if bitrev:
        want = want[_bitrev(log_n)]
    assert torch.equal(dst[4:4 + words], want.reshape(-1))
    assert (dst[:4] == -1).all() and (dst[4 + words:] == -1).all()
    assert ctx.check_device_error() == 0
