"""Which kernels run on either side of rules that the value tests cross without
looking: natural-order expansions from their smallest size on, the pair form of
CM31, and warp-owned M31 expansions."""
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


def _kernels(ctx, call):
    s = torch.cuda.current_stream().cuda_stream
    call(s)  # builds the tables
    ctx.kernel_timing(True)
    call(s)
    torch.cuda.synchronize()
    names = list(ctx.kernel_times())
    ctx.kernel_timing(False)
    return names


def _buf(words, offset=0):
    return torch.zeros(words + 8, dtype=torch.int32, device="cuda")[offset:]


@pytest.mark.parametrize("log_n,batch", [(13, 1), (13, 2), (13, 149), (14, 1)])
def test_natural_order(ctx, log_n, batch):
    lde = sfntt.CosetLdeBatch(ctx, natural=True)
    a, b = _buf(batch << log_n), _buf(batch << (log_n + 1))
    names = _kernels(ctx, lambda s: lde.execute_dev(a.data_ptr(), b.data_ptr(), log_n, batch, 1, stream=s))
    assert any(k.endswith("_lde_expand_tma_C12n") for k in names) and not any("bitrev" in k for k in names), names


@pytest.mark.parametrize("log_n,batch,offset,pairs", [(16, 24, 0, True), (12, 1, 0, True), (20, 2, 0, True),
                                                      (16, 24, 2, False), (4, 64, 0, False)])
def test_cm31(ctx, log_n, batch, offset, pairs):
    be = sfntt.Cm31Ntt(ctx)
    be.prepare(log_n, batch)
    a = _buf(2 * batch << log_n, offset)
    names = _kernels(ctx, lambda s: be.forward_dev(a.data_ptr(), log_n, batch, s))
    assert any("split" in k for k in names) != pairs, names


@pytest.mark.parametrize("log_n,batch,added,warp", [(16, 56, 1, True), (16, 55, 1, False), (16, 56, 2, True),
                                                    (16, 56, 3, False), (20, 4, 1, True)])
def test_m31_expansion(ctx, log_n, batch, added, warp):
    lde = sfntt.M31Lde(ctx)
    a, b = _buf(batch << log_n), _buf(batch << (log_n + added))
    names = _kernels(ctx, lambda s: lde.execute_dev(a.data_ptr(), b.data_ptr(), log_n, batch, added, s))
    assert ("m31_lde_expand_warp_S8" in names) == warp, names
