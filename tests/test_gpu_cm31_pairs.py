"""CM31 transforms on interleaved words: every layer count of the contiguous
pass, one and two strided passes above it, batches around whole tiles and around
the staging rule (16 columns), and buffers that fall back to the planes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

SHAPES = [(4, 3), (5, 4096), (5, 4097), (6, 2049), (7, 1025), (8, 511), (9, 257), (10, 129), (11, 65), (11, 3), (12, 1),
          (12, 15), (12, 16), (12, 17), (13, 2), (13, 16), (14, 3), (14, 17), (15, 2), (16, 1), (16, 18), (17, 1), (18, 2),
          (19, 1), (20, 1), (21, 1)]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("log_n,batch", SHAPES)
@pytest.mark.parametrize("offset", [0, 2])  # words: 16- and 8-byte aligned
def test_pairs(ctx, log_n, batch, offset):
    words = 2 * batch << log_n
    x = O.lcg(words, 7 + log_n + batch, O.M31_P)
    e = sfntt.Cm31Ntt(ctx)
    e.prepare(log_n, batch)
    buf = torch.full((words + 8,), 5, dtype=torch.int32, device="cuda")
    data = buf[offset:offset + words]
    data.copy_(torch.from_numpy(x.view(np.int32)))
    stream = torch.cuda.current_stream().cuda_stream
    e.forward_dev(data.data_ptr(), log_n, batch, stream)
    n2 = 2 << log_n
    got = data.cpu().numpy().view(np.uint32)
    for c in sorted({0, batch // 2, batch - 1}):
        assert np.array_equal(got[c * n2:(c + 1) * n2], O.cm31_ntt(x[c * n2:(c + 1) * n2], log_n, 1)), c
    e.inverse_dev(data.data_ptr(), log_n, batch, stream)
    assert np.array_equal(data.cpu().numpy().view(np.uint32), x)
    assert (buf[:offset] == 5).all() and (buf[offset + words:] == 5).all()
    assert ctx.check_device_error() == 0
