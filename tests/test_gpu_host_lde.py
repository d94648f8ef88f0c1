"""Host-buffer LDE: one and several chunks, outputs below and above the copier's
threshold and larger than its ring, pageable and pinned buffers, a copier reused
across calls, and two contexts on two threads."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import sfntt
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, log_n, batch, added, seed, pinned=False):
    x = O.lcg(batch << log_n, seed, O.BB_P, monty=True)
    lde = sfntt.CosetLdeBatch(ctx)
    if pinned:
        src, dst = ctx.pinned(x.size), ctx.pinned(x.size << added)
        src.array[:] = x
        got = lde.execute(src.array, log_n, batch, added, out=dst.array).data.copy()
        src.free()
        dst.free()
    else:
        got = lde.execute(x, log_n, batch, added).data
    n, n_ext = 1 << log_n, 1 << (log_n + added)
    for c in sorted({0, 1 % batch, batch // 2, batch - 1}):
        assert np.array_equal(got[c * n_ext:(c + 1) * n_ext], O.bb_coset_lde(x[c * n:(c + 1) * n], log_n, 1, added)), c
    return got


SHAPES = [(5, 1, 1), (8, 3, 2), (12, 63, 1), (12, 64, 1), (14, 40, 1), (16, 33, 1), (18, 24, 1), (20, 3, 2)]


@pytest.mark.parametrize("log_n,batch,added", SHAPES)
def test_pageable_equals_pinned(log_n, batch, added):
    ctx = sfntt.default_context(0)
    a = _check(ctx, log_n, batch, added, 5 + log_n)
    b = _check(ctx, log_n, batch, added, 5 + log_n, pinned=True)
    assert np.array_equal(a, b)


def test_context_comes_and_goes():
    for _ in range(3):
        c = sfntt.Context(0)
        for shape in SHAPES[3:6]:
            _check(c, *shape, 77)
        c.close()


def test_two_contexts_on_two_threads():
    bad = []

    def work(seed):
        try:
            c = sfntt.Context(0)
            for i, shape in enumerate(SHAPES * 2):
                _check(c, *shape, seed + i)
            c.close()
        except Exception as e:  # reported by the main thread
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in (100, 200)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
