"""BabyBear / KoalaBear expansions of long columns: paired output blocks stored
from registers (one column at a time) with per-position twiddles read from memory
and staged, chunk changes inside a CTA's range, and two columns at a time with
even and odd batches, one and several rounds, and the grids either side."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import sfntt  # noqa: E402
from oracle import oracle as O  # noqa: E402

ONE = [(15, 5, 1), (16, 3, 2), (16, 1, 3), (15, 15, 4),  # twiddles from memory
       (14, 76, 1), (15, 16, 1), (15, 17, 1), (16, 33, 1), (17, 17, 1),  # staged, 2x
       (16, 40, 2), (15, 60, 2), (15, 24, 3), (18, 20, 1)]
TWO = [(14, 75, 3), (14, 100, 4), (14, 147, 3), (14, 148, 3), (15, 60, 4), (15, 61, 3), (16, 21, 3), (16, 33, 4),
       (17, 16, 3), (17, 31, 3), (18, 18, 3)]


@pytest.fixture(scope="module")
def ctx():
    c = sfntt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("log_n,batch,added,two", [(*s, False) for s in ONE] + [(*s, True) for s in TWO])
@pytest.mark.parametrize("field", ["bb", "kb"])
def test_expansion(ctx, field, log_n, batch, added, two):
    p = O.KB_P if field == "kb" else O.BB_P
    x = O.lcg(batch << log_n, 41 + log_n, p, monty=True)
    x[::97] = p - 1
    shift = 777 if batch & 1 else 0
    ref = (O.kb_coset_lde if field == "kb" else O.bb_coset_lde)(x, log_n, batch, added, shift_monty=shift, threads=8)
    lde = (sfntt.KbCosetLdeBatch if field == "kb" else sfntt.CosetLdeBatch)(ctx)
    d_in = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.full(((batch << (log_n + added)) + 64,), 99, dtype=torch.int32, device="cuda")
    ctx.kernel_timing(True)
    for _ in range(2):  # the second call finds every table resident
        out[:-64].fill_(-1)
        lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, batch, added, shift_monty=shift,
                        stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (out[-64:] == 99).all()
        assert np.array_equal(out[:-64].cpu().numpy().view(np.uint32), ref)
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    assert any(k.endswith("S8cc") for k in names) == two, names
    if not two:
        assert any("_expand_tma_S8" in k for k in names), names


def _rev(k):
    i = np.arange(1 << k)
    r = np.zeros_like(i)
    for _ in range(k):
        r, i = (r << 1) | (i & 1), i >> 1
    return r


@pytest.mark.parametrize("log_n,batch", [(13, 1), (13, 2), (13, 149), (14, 37), (14, 149), (15, 3), (16, 55), (18, 5), (20, 2)])
@pytest.mark.parametrize("field", ["bb", "kb"])
def test_natural_order(ctx, field, log_n, batch):
    """Natural-order 2x expansion: one tile, one tile per CTA and one more, several per CTA."""
    p = O.KB_P if field == "kb" else O.BB_P
    x = O.lcg(batch << log_n, 53 + log_n, p, monty=True)
    x[::89] = p - 1
    shift = 999 if batch & 1 else 0
    br = np.ascontiguousarray(x.reshape(batch, -1)[:, _rev(log_n)]).reshape(-1)
    ref = (O.kb_coset_lde if field == "kb" else O.bb_coset_lde)(br, log_n, batch, 1, shift_monty=shift, threads=8)
    ref = ref.reshape(batch, -1)[:, _rev(log_n + 1)].reshape(-1)
    lde = (sfntt.KbCosetLdeBatch if field == "kb" else sfntt.CosetLdeBatch)(ctx, natural=True)
    d_in = torch.from_numpy(x.view(np.int32).copy()).cuda()
    out = torch.full(((batch << (log_n + 1)) + 64,), 99, dtype=torch.int32, device="cuda")
    ctx.kernel_timing(True)
    for _ in range(2):
        out[:-64].fill_(-1)
        lde.execute_dev(d_in.data_ptr(), out.data_ptr(), log_n, batch, 1, shift_monty=shift,
                        stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (out[-64:] == 99).all()
        assert np.array_equal(out[:-64].cpu().numpy().view(np.uint32), ref)
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    assert log_n == 13 or any(k.endswith("_lde_expand_tma_C12n") for k in names), names
