"""Representative workloads of the library, each one pass through its public calls.

A case is a dict of plain values; `kind` selects the family:

  ntt     a batch of columns, forward in place on one buffer, inverse on another
  cm31    the same over CM31 pairs, then the pointwise product of the two
  lde     a coset LDE (BabyBear, KoalaBear) or blow-up (M31, circle) of a batch
  commit  the input of a Merkle commitment: natural-order coset LDE with the
          shift 31, row-major rows, canonical words
  graph   an uneven batch of LDEs of two fields, replayed as one CUDA graph
  host    a coset LDE called on host arrays

Sizes: log_n points per column, batch columns, added blow-up bits.
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import torch

PKG = str(Path(__file__).resolve().parents[1] / "small-field-metal-ntt_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import sfntt  # noqa: E402

PRIMES = {"m31": sfntt.M31_P, "circle": sfntt.M31_P, "bb": sfntt.BB_P, "kb": sfntt.KB_P}
GENERATORS = {"bb": 31, "kb": 3}
BACKENDS = {"m31": sfntt.CudaCtGsR4, "bb": sfntt.BbCudaCtGsR4, "kb": sfntt.KbCudaCtGsR4}
MONTY_R = 1 << 32
COMMIT_SHIFT = 31


def listed():
    return [
        # a polynomial of a small circuit or a test: launches and the call are the cost
        {"name": "ntt_bb_2^10_x1", "kind": "ntt", "field": "bb", "log_n": 10, "batch": 1},
        # the reference's single-column Circle NTT benchmark size
        {"name": "ntt_m31_2^16_x1", "kind": "ntt", "field": "m31", "log_n": 16, "batch": 1},
        # the largest single column of the reference's benchmark
        {"name": "ntt_bb_2^24_x1", "kind": "ntt", "field": "bb", "log_n": 24, "batch": 1},
        # thousands of short transforms (lattice-style batches), a count that fills no tile evenly
        {"name": "ntt_bb_2^9_x20001", "kind": "ntt", "field": "bb", "log_n": 9, "batch": 20001},
        # an ordinary trace: an odd number of mid-sized columns
        {"name": "ntt_kb_2^17_x37", "kind": "ntt", "field": "kb", "log_n": 17, "batch": 37},
        # extension-field columns: both transforms and a product
        {"name": "cm31_2^16_x24", "kind": "cm31", "log_n": 16, "batch": 24},
        # the headline: the reference's batched coset LDE
        {"name": "lde_bb_2^20_x256_2x", "kind": "lde", "field": "bb", "log_n": 20, "batch": 256, "added": 1},
        # a short trace at a larger blow-up (a recursion layer, a lookup table)
        {"name": "lde_bb_2^11_x200_4x", "kind": "lde", "field": "bb", "log_n": 11, "batch": 200, "added": 2},
        # the Stwo-style circle LDE of an odd number of long columns
        {"name": "lde_circle_2^20_x61_2x", "kind": "lde", "field": "circle", "log_n": 20, "batch": 61, "added": 1},
        # the commitment path of a prover: extension, row-major rows, canonical words
        {"name": "commit_bb_2^18_x100_2x", "kind": "commit", "field": "bb", "log_n": 18, "batch": 100, "added": 1},
        # many polynomials of uneven sizes, both fields, in one launch
        {"name": "graph_uneven_24", "kind": "graph", "items": 24, "mix": 7, "log_lo": 12, "log_hi": 19, "cols": 64},
        # the drop-in call: host memory in, host memory out
        {"name": "host_lde_bb_2^14_x40_2x", "kind": "host", "field": "bb", "log_n": 14, "batch": 40, "added": 1},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "ntt", "cm31", "lde", "lde", "lde", "commit", "graph", "host"])
    if kind == "ntt":
        log_n = rng.randint(6, 24)
        return {"kind": kind, "field": rng.choice(["m31", "bb", "kb"]), "log_n": log_n,
                "batch": _log_uniform(rng, 1, max(1, (1 << 26) >> log_n))}
    if kind == "cm31":
        log_n = rng.randint(8, 20)
        return {"kind": kind, "log_n": log_n, "batch": _log_uniform(rng, 1, max(1, (1 << 23) >> log_n))}
    if kind == "lde":
        log_n, added = rng.randint(8, 21), rng.randint(1, 3)
        return {"kind": kind, "field": rng.choice(["bb", "bb", "kb", "m31", "circle"]), "log_n": log_n,
                "batch": _log_uniform(rng, 1, max(1, min(500, (1 << 28) >> (log_n + added)))), "added": added}
    if kind == "commit":
        log_n = rng.randint(12, 20)
        return {"kind": kind, "field": rng.choice(["bb", "kb"]), "log_n": log_n,
                "batch": _log_uniform(rng, 4, max(4, min(300, (1 << 26) >> log_n))), "added": 1}
    if kind == "graph":
        lo = rng.randint(12, 14)
        return {"kind": kind, "items": rng.randint(8, 32), "mix": rng.randint(1, 10000), "log_lo": lo,
                "log_hi": lo + rng.randint(3, 5), "cols": rng.randint(16, 64)}
    log_n = rng.randint(8, 18)
    return {"kind": kind, "field": rng.choice(["bb", "kb"]), "log_n": log_n,
            "batch": _log_uniform(rng, 1, max(1, min(300, (1 << 22) >> log_n))), "added": rng.randint(1, 2)}


# ------------------------------------------------------------------ inputs ---
def _words(count, p, gen):
    """Uniform field elements (canonical M31, Montgomery BabyBear / KoalaBear)."""
    return torch.randint(0, p, (count,), dtype=torch.int32, device="cuda", generator=gen)


def _graph_items(case):
    return sfntt.uneven_workload(case["items"], seed=case["mix"], log_n_range=(case["log_lo"], case["log_hi"]),
                                 cols_range=(1, case["cols"]))


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "graph":
        names = {sfntt.FIELD_M31: "m31", sfntt.FIELD_BABYBEAR: "bb"}
        return [_words(it["batch"] << it["log_n"], PRIMES[names[it["field"]]], gen) for it in _graph_items(case)]
    total = case["batch"] << case["log_n"]
    if kind == "ntt":
        return [_words(total, PRIMES[case["field"]], gen) for _ in range(2)]
    if kind == "cm31":
        return [_words(2 * total, sfntt.M31_P, gen) for _ in range(2)]
    return [_words(total, PRIMES[case["field"]], gen)]


def _commit_shift(field):
    return COMMIT_SHIFT * MONTY_R % PRIMES[field]


def prepare(case, seed):
    ctx = sfntt.default_context(0)
    xs = _inputs(case, seed)
    s = {"case": case, "ctx": ctx, "xs": xs}
    kind = case["kind"]
    if kind == "ntt":
        s["backend"] = BACKENDS[case["field"]](ctx)
        ctx.prepare(s["backend"].FIELD, case["log_n"])
    elif kind == "cm31":
        s["backend"] = sfntt.Cm31Ntt(ctx)
        s["backend"].prepare(case["log_n"], case["batch"])
        s["out"] = torch.empty_like(xs[0])
    elif kind in ("lde", "commit"):
        field, words = case["field"], case["batch"] << (case["log_n"] + case["added"])
        s["out"] = torch.empty(words, dtype=torch.int32, device="cuda")
        if field == "circle":
            s["lde"] = sfntt.CircleLde(ctx)
            s["lde"].prepare(case["log_n"], case["added"])
        elif field == "m31":
            s["lde"] = sfntt.M31Lde(ctx)
            ctx.prepare_lde(sfntt.FIELD_M31, case["log_n"], case["added"])
        else:
            cls = sfntt.KbCosetLdeBatch if field == "kb" else sfntt.CosetLdeBatch
            s["lde"] = cls(ctx, natural=kind == "commit")
            ctx.prepare_lde(cls.FIELD, case["log_n"], case["added"], _commit_shift(field) if kind == "commit" else 0)
        if kind == "commit":
            s["rows"] = torch.empty(words, dtype=torch.int32, device="cuda")
    elif kind == "graph":
        items = _graph_items(case)
        s["outs"] = [torch.empty(it["batch"] << (it["log_n"] + it["added_bits"]), dtype=torch.int32, device="cuda")
                     for it in items]
        for it, x, o in zip(items, xs, s["outs"]):
            it["d_in"], it["d_out"] = x.data_ptr(), o.data_ptr()
        s["batch"] = sfntt.LdeBatch(ctx, items)
        s["batch"].prepare()
        s["graph"] = s["batch"].graph()
    else:
        s["lde"] = (sfntt.KbCosetLdeBatch if case["field"] == "kb" else sfntt.CosetLdeBatch)(ctx)
        s["host"] = xs[0].cpu().numpy().view(np.uint32)
    return s


# -------------------------------------------------------------------- run ---
def run(s):
    case, xs = s["case"], s["xs"]
    kind = case["kind"]
    if kind == "host":
        return s["lde"].execute(s["host"], case["log_n"], case["batch"], case["added"]).data.view(np.int32)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "graph":
        s["graph"].launch(stream)
        return s["outs"]
    log_n, batch = case["log_n"], case["batch"]
    if kind == "ntt":
        s["backend"].forward_dev(xs[0].data_ptr(), log_n, batch, stream)
        s["backend"].inverse_dev(xs[1].data_ptr(), log_n, batch, stream)
        return xs
    if kind == "cm31":
        s["backend"].forward_dev(xs[0].data_ptr(), log_n, batch, stream)
        s["backend"].inverse_dev(xs[1].data_ptr(), log_n, batch, stream)
        s["backend"].mul_dev(xs[0].data_ptr(), xs[1].data_ptr(), s["out"].data_ptr(), batch << log_n, stream)
        return [xs[0], xs[1], s["out"]]
    if kind == "lde":
        if case["field"] in ("m31", "circle"):
            s["lde"].execute_dev(xs[0].data_ptr(), s["out"].data_ptr(), log_n, batch, case["added"], stream)
        else:
            s["lde"].execute_dev(xs[0].data_ptr(), s["out"].data_ptr(), log_n, batch, case["added"], 0, stream)
        return s["out"]
    s["lde"].execute_dev(xs[0].data_ptr(), s["out"].data_ptr(), log_n, batch, case["added"],
                         _commit_shift(case["field"]), stream)
    sfntt.layout_dev(s["ctx"], s["out"].data_ptr(), s["rows"].data_ptr(), log_n + case["added"], batch,
                     sfntt.LAYOUT_ROW_MAJOR, stream)
    sfntt.convert_monty_dev(s["ctx"], s["lde"].FIELD, s["rows"].data_ptr(), s["rows"].numel(), False, stream)
    return s["rows"]


# ------------------------------------------------------------------- work ---
def _ntt_ops(points, log_n):
    """Modular operations of the butterflies: a product, a sum and a difference each."""
    return 3 * points // 2 * log_n


def _lde_work(log_n, batch, added):
    n, n_ext = batch << log_n, batch << (log_n + added)
    # inverse layers, one factor per output (scaling, shift and the layers over
    # zeros), then the remaining forward layers of every block
    return 4 * (n + n_ext), _ntt_ops(n, log_n) + n_ext + _ntt_ops(n_ext, log_n)


def work(case):
    kind = case["kind"]
    if kind == "graph":
        parts = [_lde_work(it["log_n"], it["batch"], it["added_bits"]) for it in _graph_items(case)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    log_n, batch = case["log_n"], case["batch"]
    points = batch << log_n
    if kind == "ntt":
        return {"bytes": 2 * 8 * points, "flops": 2 * _ntt_ops(points, log_n)}
    if kind == "cm31":
        return {"bytes": 8 * points * 5, "flops": 2 * _ntt_ops(2 * points, log_n) + 6 * points}
    b, f = _lde_work(log_n, batch, case["added"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact ---
# Plain 64-bit integer forms of the transforms, layer by layer.
def _powers(base, count, p, start=1):
    t = torch.tensor([start % p], dtype=torch.int64, device="cuda")
    step = base % p
    while t.numel() < count:
        t = torch.cat([t, t * step % p])
        step = step * step % p
    return t[:count]


def _root(field, log_n):
    p = PRIMES[field]
    return pow(GENERATORS[field], (p - 1) >> log_n, p)


def _rev(bits):
    i = torch.arange(1 << bits, dtype=torch.int64, device="cuda")
    r = torch.zeros_like(i)
    for b in range(bits):
        r = (r << 1) | ((i >> b) & 1)
    return r


def _monty_forward(x, field, log_n):
    """x: [columns, n], natural order in, bit-reversed order out."""
    p = PRIMES[field]
    for layer in range(log_n - 1, -1, -1):
        w = _powers(_root(field, layer + 1), 1 << layer, p)
        v = x.view(x.shape[0], -1, 2, 1 << layer)
        a, b = v[:, :, 0], v[:, :, 1]
        x = torch.stack([(a + b) % p, (a - b + p) * w % p], dim=2).reshape(x.shape[0], -1)
    return x


def _monty_inverse(x, field, log_n):
    p = PRIMES[field]
    for layer in range(log_n):
        w = _powers(pow(_root(field, layer + 1), p - 2, p), 1 << layer, p)
        v = x.view(x.shape[0], -1, 2, 1 << layer)
        a, b = v[:, :, 0], v[:, :, 1] * w % p
        x = torch.stack([(a + b) % p, (a - b + p) % p], dim=2).reshape(x.shape[0], -1)
    return x * pow(1 << log_n, p - 2, p) % p


def _circle_add(a, b):
    p = sfntt.M31_P
    return (a[0] * b[0] % p - a[1] * b[1] % p) % p, (a[0] * b[1] % p + a[1] * b[0] % p) % p


def _circle_gen(log_size):
    g = (2, 1268011823)
    for _ in range(31 - log_size):
        g = _circle_add(g, g)
    return g


def _circle_coset(first, step, log_count):
    """Points first + i step, i < 2^log_count, in bit-reversed order of i."""
    x = torch.tensor([first[0]], dtype=torch.int64, device="cuda")
    y = torch.tensor([first[1]], dtype=torch.int64, device="cuda")
    for _ in range(log_count):
        x2, y2 = _circle_add((x, y), step)
        x, y = torch.cat([x, x2]), torch.cat([y, y2])
        step = _circle_add(step, step)
    r = _rev(log_count)
    return x[r], y[r]


def _m31_twiddles(log_n, canonic):
    """Per layer L the factors of its 2^(log_n - 1 - L) blocks."""
    out = []
    if canonic:
        g = _circle_gen(log_n + 1)
        step = _circle_add(g, g)
        for layer in range(log_n):
            if layer == 0:
                out.append(_circle_coset(g, _circle_add(step, step), log_n - 1)[1])
                continue
            out.append(_circle_coset(g, _circle_add(step, step), log_n - 1 - layer)[0])
            g, step = _circle_add(g, g), _circle_add(step, step)
        return out
    first, step = _circle_gen(log_n + 1), _circle_gen(log_n)
    for layer in range(log_n):
        pts = _circle_coset(first, step, log_n - 1 - layer)
        out.append(pts[1] if layer == log_n - 1 else pts[0])
        first, step = _circle_add(first, first), _circle_add(step, step)
    return out


def _m31_inv(x):
    p, r, e = sfntt.M31_P, torch.ones_like(x), sfntt.M31_P - 2
    while e:
        if e & 1:
            r = r * x % p
        x = x * x % p
        e >>= 1
    return r


def _m31_forward(x, tw, log_n):
    p = sfntt.M31_P
    for layer in range(log_n - 1, -1, -1):
        v = x.view(x.shape[0], -1, 2, 1 << layer)
        a, b = v[:, :, 0], v[:, :, 1] * tw[layer][None, :, None] % p
        x = torch.stack([(a + b) % p, (a - b + p) % p], dim=2).reshape(x.shape[0], -1)
    return x


def _m31_inverse(x, itw, log_n):
    p = sfntt.M31_P
    for layer in range(log_n):
        v = x.view(x.shape[0], -1, 2, 1 << layer)
        a, b = v[:, :, 0], v[:, :, 1]
        x = torch.stack([(a + b) % p, (a - b + p) * itw[layer][None, :, None] % p], dim=2).reshape(x.shape[0], -1)
    return x * pow(1 << log_n, p - 2, p) % p


def _by_columns(x, n, n_out, fn):
    """fn over chunks of columns of a SoA batch (64-bit copies of a chunk stay small)."""
    cols = x.numel() // n
    out = torch.empty(cols * n_out, dtype=torch.int32, device="cuda")
    step = max(1, (1 << 25) // max(n, n_out))
    for c in range(0, cols, step):
        e = min(cols, c + step)
        out[c * n_out:e * n_out] = fn(x[c * n:e * n].view(-1, n).to(torch.int64)).reshape(-1).to(torch.int32)
    return out


def _ntt_exact(x, field, log_n, inverse):
    if field in GENERATORS:
        fn = _monty_inverse if inverse else _monty_forward
        return _by_columns(x, 1 << log_n, 1 << log_n, lambda v: fn(v, field, log_n))
    tw = _m31_twiddles(log_n, False)
    if inverse:
        itw = [_m31_inv(t) for t in tw]
        return _by_columns(x, 1 << log_n, 1 << log_n, lambda v: _m31_inverse(v, itw, log_n))
    return _by_columns(x, 1 << log_n, 1 << log_n, lambda v: _m31_forward(v, tw, log_n))


def _lde_exact(x, field, log_n, added, shift=None, natural=False):
    n, n_ext, log_ext = 1 << log_n, 1 << (log_n + added), log_n + added
    p = PRIMES[field]
    if field in GENERATORS:
        powers = _powers(_root(field, log_ext + 1) if shift is None else shift, n, p)
        rev_in, rev_out = _rev(log_n), _rev(log_ext)

        def extend(v):
            v = _monty_inverse(v[:, rev_in] if natural else v, field, log_n) * powers % p
            v = _monty_forward(torch.nn.functional.pad(v, (0, n_ext - n)), field, log_ext)
            return v[:, rev_out] if natural else v
    else:
        itw = [_m31_inv(t) for t in _m31_twiddles(log_n, field == "circle")]
        tw = _m31_twiddles(log_ext, field == "circle")

        def extend(v):
            return _m31_forward(torch.nn.functional.pad(_m31_inverse(v, itw, log_n), (0, n_ext - n)), tw, log_ext)
    return _by_columns(x, n, n_ext, extend)


def exact(case, seed):
    xs = _inputs(case, seed)
    kind = case["kind"]
    if kind == "graph":
        names = {sfntt.FIELD_M31: "m31", sfntt.FIELD_BABYBEAR: "bb"}
        return [_lde_exact(x, names[it["field"]], it["log_n"], it["added_bits"])
                for it, x in zip(_graph_items(case), xs)]
    log_n, batch = case["log_n"], case["batch"]
    if kind == "ntt":
        return [_ntt_exact(xs[0], case["field"], log_n, False), _ntt_exact(xs[1], case["field"], log_n, True)]
    if kind == "cm31":
        def pairs(x, inverse):
            planes = x.view(-1, 2).t().contiguous().view(-1)
            return _ntt_exact(planes, "m31", log_n, inverse).view(2, -1).t().contiguous().view(-1)
        a, b = pairs(xs[0], False), pairs(xs[1], True)
        p, u, v = sfntt.M31_P, a.view(-1, 2).to(torch.int64), b.view(-1, 2).to(torch.int64)
        re = (u[:, 0] * v[:, 0] % p - u[:, 1] * v[:, 1] % p) % p
        im = (u[:, 0] * v[:, 1] % p + u[:, 1] * v[:, 0] % p) % p
        return [a, b, torch.stack([re, im], dim=1).view(-1).to(torch.int32)]
    if kind == "commit":
        field = case["field"]
        p = PRIMES[field]
        rows = _lde_exact(xs[0], field, log_n, case["added"], COMMIT_SHIFT, natural=True).view(batch, -1).t()
        r_inv = pow(MONTY_R, p - 2, p)
        return (rows.contiguous().view(-1).to(torch.int64) * r_inv % p).to(torch.int32)
    y = _lde_exact(xs[0], case["field"], log_n, case["added"])
    return y.cpu().numpy() if kind == "host" else y
