"""Which engine a batch of short columns takes when its last tile stays part empty:
either side of the lines, by field, size and direction."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

BACKENDS = {"bb": (sfntt.BbCudaCtGsR4, O.BB_P, O.bb_forward, O.bb_inverse),
            "m31": (sfntt.CudaCtGsR4, O.M31_P, O.m31_forward, O.m31_inverse)}
# field, log_n, batch, forward on the tile engine, inverse
LINES = [("m31", 8, (3 << 9) - 1, False, False), ("m31", 8, (3 << 9) + 1, True, True),
         ("m31", 9, (9 << 7) - 1, False, False), ("m31", 9, (9 << 7) + 1, True, True),
         ("m31", 11, (3 << 6) - 1, False, False), ("m31", 11, (3 << 6) + 1, True, True),
         ("m31", 7, (1 << 11) + 1, True, True), ("m31", 10, (1 << 8), True, True),  # whole tiles
         ("bb", 9, (1 << 9) + 1, True, False), ("bb", 9, (3 << 8) - 1, True, False), ("bb", 9, (3 << 8) + 1, True, True),
         ("bb", 8, (1 << 10) + 1, True, True), ("bb", 8, (1 << 10) - 1, False, False), ("m31", 12, 3, True, True)]


@pytest.mark.parametrize("field,log_n,batch,f_tma,i_tma", LINES)
def test_engine(field, log_n, batch, f_tma, i_tma):
    cls, p, fwd, inv = BACKENDS[field]
    ctx = sfntt.default_context(0)
    n = 1 << log_n
    x = O.lcg(batch * n, 9 + log_n, p, monty=field != "m31")
    b = cls(ctx)
    for run, ref, tma in ((b.forward_dev, fwd, f_tma), (b.inverse_dev, inv, i_tma)):
        d = torch.from_numpy(x.view(np.int32).copy()).cuda()
        ctx.kernel_timing(True)
        run(d.data_ptr(), log_n, batch, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        names = list(ctx.kernel_times())
        ctx.kernel_timing(False)
        assert any("_tma_C" in k for k in names) == tma, names
        got = d.cpu().numpy().view(np.uint32)
        for c in (0, batch // 2, batch - 1):
            assert np.array_equal(got[c * n:(c + 1) * n], ref(x[c * n:(c + 1) * n])), c
