"""Batches of short columns that do not fill their last tile: every column
length below a tile, one column more and less than whole tiles, a last tile
that ends inside its first half, and the sizes where the rule changes engine."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

BACKENDS = {"bb": (sfntt.BbCudaCtGsR4, O.BB_P, O.bb_forward, O.bb_inverse),
            "kb": (sfntt.KbCudaCtGsR4, O.KB_P, O.kb_forward, O.kb_inverse),
            "m31": (sfntt.CudaCtGsR4, O.M31_P, O.m31_forward, O.m31_inverse)}
SHAPES = [(log_n, (1 << (18 - log_n)) + extra) for log_n in range(5, 13) for extra in (-1, 1)]
SHAPES += [(log_n, (3 << (18 - log_n)) + (1 << (12 - log_n)) + 1) for log_n in (5, 8, 11)] + [(12, 3), (12, 1), (4, 70001)]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("field", sorted(BACKENDS))
@pytest.mark.parametrize("log_n,batch", SHAPES)
def test_ragged_batch(ctx, field, log_n, batch):
    cls, p, fwd, inv = BACKENDS[field]
    n = 1 << log_n
    x = O.lcg(batch * n, 3 + log_n + batch, p, monty=field != "m31")
    buf = torch.full((batch * n + 64,), 12345, dtype=torch.int32, device="cuda")
    data = buf[:batch * n]
    data.copy_(torch.from_numpy(x.view(np.int32)))
    b = cls(ctx)
    stream = torch.cuda.current_stream().cuda_stream
    b.forward_dev(data.data_ptr(), log_n, batch, stream)
    got = data.cpu().numpy().view(np.uint32)
    cols = sorted({0, 1, batch // 2, batch - 2, batch - 1} & set(range(batch)))
    for c in cols:
        assert np.array_equal(got[c * n:(c + 1) * n], fwd(x[c * n:(c + 1) * n])), c
    b.inverse_dev(data.data_ptr(), log_n, batch, stream)
    assert np.array_equal(data.cpu().numpy().view(np.uint32), x)
    data.copy_(torch.from_numpy(x.view(np.int32)))
    b.inverse_dev(data.data_ptr(), log_n, batch, stream)
    got = data.cpu().numpy().view(np.uint32)
    for c in cols:
        assert np.array_equal(got[c * n:(c + 1) * n], inv(x[c * n:(c + 1) * n])), c
    assert (buf[batch * n:] == 12345).all()
    assert ctx.check_device_error() == 0
