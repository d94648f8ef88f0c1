"""Element-wise maps around the size where they change from words to 16-byte
vectors, aligned and not, in place and over two arrays."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

SIZES = [1, 4095, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 18) + 4099]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("offset", [0, 1])
def test_conversion(n, offset):
    ctx = sfntt.default_context(0)
    x = O.lcg(n, 3 + n, O.BB_P)
    buf = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
    buf[offset:offset + n] = torch.from_numpy(x.view(np.int32))
    s = torch.cuda.current_stream().cuda_stream
    ctx.kernel_timing(True)
    sfntt.convert_monty_dev(ctx, sfntt.FIELD_BABYBEAR, buf.data_ptr() + 4 * offset, n, True, s)
    torch.cuda.synchronize()
    # blocks of 16 KiB only where they reach every SM
    assert list(ctx.kernel_times()) == ["to_monty_vec" if offset == 0 and n > 1 << 18 else "to_monty"]
    ctx.kernel_timing(False)
    got = buf.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[offset:offset + n].astype(np.uint64), (x.astype(np.uint64) << np.uint64(32)) % np.uint64(O.BB_P))
    sfntt.convert_monty_dev(ctx, sfntt.FIELD_BABYBEAR, buf.data_ptr() + 4 * offset, n, False, s)
    got = buf.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[offset:offset + n], x)
    assert (got[:offset] == 7).all() and (got[offset + n:] == 7).all()


@pytest.mark.parametrize("n", SIZES)
def test_product(n):
    a, b = O.lcg(n, 5, O.M31_P), O.lcg(n, 6, O.M31_P)
    out = np.empty(n, dtype=np.uint32)
    sfntt.CudaCtGsR4(sfntt.default_context(0)).pointwise_mul(a, b, out)
    assert np.array_equal(out.astype(np.uint64), a.astype(np.uint64) * b % np.uint64(O.M31_P))
