"""Element-wise kernels at the edges of their vector form: tails of 0..3 words,
one block more or less, and buffers that are not 16-byte aligned."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

FIELDS = {sfntt.FIELD_BABYBEAR: sfntt.BB_P, sfntt.FIELD_KOALABEAR: sfntt.KB_P}
SIZES = [1, 3, 4, 7, 4095, 4096, 4097, 4098, 4099, 3 * 4096 + 2, 1 << 17]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("field", sorted(FIELDS))
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_monty_conversion(ctx, field, offset, n):
    p = FIELDS[field]
    x = O.lcg(n, 11 + n, p)
    buf = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(x.view(np.int32)).cuda()
    ptr = buf.data_ptr() + 4 * offset
    sfntt.convert_monty_dev(ctx, field, ptr, n, True)
    torch.cuda.synchronize()
    got = buf.cpu().numpy().view(np.uint32)
    want = (x.astype(np.uint64) << np.uint64(32)) % np.uint64(p)
    assert np.array_equal(got[offset:offset + n], want.astype(np.uint32))
    assert (got[:offset] == 7).all() and (got[offset + n:] == 7).all()
    sfntt.convert_monty_dev(ctx, field, ptr, n, False)
    torch.cuda.synchronize()
    assert np.array_equal(buf.cpu().numpy().view(np.uint32)[offset:offset + n], x)


@pytest.mark.parametrize("cls,p,mul", [(sfntt.BbCudaCtGsR4, sfntt.BB_P, "bb"), (sfntt.CudaCtGsR4, sfntt.M31_P, "m31")])
@pytest.mark.parametrize("n", SIZES)
def test_pointwise(ctx, cls, p, mul, n):
    a, b = O.lcg(n, 5, p), O.lcg(n, 6, p)
    out = np.empty(n, dtype=np.uint32)
    cls(ctx).pointwise_mul(a, b, out)
    prod = a.astype(object) * b.astype(object)
    if mul == "bb":
        prod = prod * pow(1 << 32, p - 2, p)
    assert np.array_equal(out, (prod % p).astype(np.uint32))
