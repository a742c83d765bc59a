"""Kernels of attention with options (csrc/attention_scored.cu) against the general ones and float64, over the forms that they
take: runs of keys that end inside a tile, windows with kept first keys, chunks, caps, sinks, biases, gates, one to five query
heads a key head."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d,heads,kv", [(128, 16, 4), (64, 8, 8), (128, 10, 2), (64, 6, 2), (128, 5, 5)])
@pytest.mark.parametrize("mask,size,keep,extra", [("causal", 0, 0, "sink"), ("window", 100, 0, "cap"), ("window", 37, 5, "bias"),
                                                  ("chunk", 64, 0, "gate"), ("window", 1, 0, "none"), ("causal", 0, 0, "cap bias gate sink")])
def test_decode_on_tensor_cores(d, heads, kv, mask, size, keep, extra):
    """Products of bfloat16 numbers are exact, weights keep 24 bits and sums are float32, so what differs from float64 is the
    rounding of the output to bfloat16 (2^-9) and float32 noise; no further off than the kernel of a lane per key."""
    from llm_rs_b200 import ops
    torch.manual_seed(d + heads + size)
    page, cached = 16, [0, 15, 16, 200, 777, 63]
    n, width = len(cached), -(-778 // page)
    q = torch.randn(n, heads * d + 8, device=DEV).bfloat16()[:, : heads * d]
    cache = torch.randn(n * width, kv, page * 2 * d, device=DEV).bfloat16()
    table = torch.randperm(n * width, device=DEV).to(torch.int32).view(n, width)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(q_start=i32(list(range(n))), cached_len=i32(cached), scratch=lambda name, f: torch.empty(f, device=DEV))
    sink = torch.randn(heads, device=DEV) if "sink" in extra else None
    bias = torch.randn(90, heads, device=DEV) if "bias" in extra else None
    gate = torch.randn(n, heads, device=DEV).bfloat16() if "gate" in extra else None
    cap, scale = (5.0 if "cap" in extra else 0.0), 0.7 / math.sqrt(d)
    want = torch.empty(n, heads, d, dtype=torch.float64, device=DEV)
    for r, c in enumerate(cached):
        keys = torch.arange(c + 1, device=DEV)
        lo = {"causal": 0, "window": max(0, c - size + 1), "chunk": c // size * size if size else 0}[mask]
        keys = keys[(keys >= lo) | (keys < keep)]
        pg = cache[table[r, keys // page].long()].double()
        at = torch.arange(len(keys), device=DEV)
        ks = pg[:, :, : page * d].unflatten(2, (page, d))[at, :, keys % page]
        vs = pg[:, :, page * d:].unflatten(2, (page, d))[at, :, keys % page]
        for h in range(heads):
            s = ks[:, h // (heads // kv)] @ q[r, h * d: (h + 1) * d].double() * scale
            s = cap * torch.tanh(s / cap) if cap else s
            if bias is not None:
                s = s + bias[(c - keys).clamp(0, 89), h].double()
            if sink is not None:
                s = torch.cat([s, sink[h].double()[None]])
            p = torch.softmax(s, 0)[: len(keys)]
            want[r, h] = p @ vs[:, h // (heads // kv)] * (torch.sigmoid(gate[r, h].double()) if gate is not None else 1.0)
    errors = []
    for generic, (runs, keys) in ((False, (13, 64)), (False, (2, 512)), (True, (7, 128))):
        out = torch.zeros(n, heads * d, device=DEV).bfloat16()
        ops.scored_generic_only(generic)
        try:
            ops.scored_decode(q, out, cache, i32(list(range(n))), n, ctx, table, runs, keys, heads, kv, d, d, page, scale, cap, sink,
                              {"causal": 0, "window": 1, "chunk": 2}[mask], size, bias=bias, keep=keep, gate=gate)
        finally:
            ops.scored_generic_only(False)
        err = (out.view(n, heads, d).double() - want).abs()
        assert bool((err <= 2.0 ** -8 * want.abs() + 1e-5).all()), (generic, runs)
        errors.append(float(err.norm() / want.norm()))
    assert max(errors[:2]) <= 1.02 * errors[2]


@pytest.mark.parametrize("generic", [False, True])
def test_decode_keeps_infinite_values(generic):
    """An infinite value of a visible key makes its channel infinite, two of opposite signs or a NaN make it NaN, on both
    kernels; other channels do not change."""
    from llm_rs_b200 import ops
    torch.manual_seed(3)
    d, heads, kv, page, cached = 64, 4, 2, 16, 99
    q = torch.randn(1, heads * d, device=DEV).bfloat16() * 0.1
    cache = torch.randn(7, kv, page * 2 * d, device=DEV).bfloat16()
    values = cache[:, :, page * d:].unflatten(2, (page, d))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table = i32([list(range(7))])
    ctx = SimpleNamespace(q_start=i32([0]), cached_len=i32([cached]), scratch=lambda name, f: torch.empty(f, device=DEV))

    def run():
        out = torch.zeros(1, heads * d, device=DEV).bfloat16()
        ops.scored_generic_only(generic)
        try:
            ops.scored_decode(q, out, cache, i32([0]), 1, ctx, table, 2, 64, heads, kv, d, d, page, 0.125, 0.0, None, 0, 0)
        finally:
            ops.scored_generic_only(False)
        return out.view(kv, heads // kv, d).float()

    before = run()
    values[2, 0, 3, 5], values[6, 0, 3, 6], values[6, 0, 4, 7] = math.inf, -math.inf, math.nan      # the last key: 99 = 6 * 16 + 3
    values[0, 1, 0, 8], values[1, 1, 1, 8] = math.inf, -math.inf
    after = run()
    assert bool((after[0, :, 5] == math.inf).all()) and bool((after[0, :, 6] == -math.inf).all())
    assert bool(after[1, :, 8].isnan().all()) and not bool(after[0, :, 7].isnan().any())      # (key 100 is not visible)
    rest = torch.ones_like(before, dtype=torch.bool)
    rest[0, :, 5], rest[0, :, 6], rest[1, :, 8] = False, False, False
    assert torch.equal(before[rest], after[rest])


def _prepared(x, heads, dk, norm, weight, inv_freq, positions, rot, pairs):
    """Heads normed and rotated in float64 by the definition."""
    x = x.double().view(-1, heads, dk)
    if norm == "whole":
        x = x / torch.sqrt((x ** 2).mean((1, 2), keepdim=True) + 1e-6) * weight.double().view(heads, dk)
    elif norm in ("unit", "shared"):
        x = x / torch.sqrt((x ** 2).mean(2, keepdim=True) + 1e-6) * (weight.double() if norm == "shared" else 1.0)
    angle = (positions.double()[:, None] * inv_freq)[:, None]
    turned = x[..., :rot].unflatten(2, (rot // 2, 2)).transpose(2, 3) if pairs else x[..., :rot].unflatten(2, (2, rot // 2))
    a, b = turned[:, :, 0], turned[:, :, 1]
    turned = torch.stack([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], 2)
    turned = (turned.transpose(2, 3) if pairs else turned).flatten(2)
    return torch.cat([turned, x[..., rot:]], 2)


@pytest.mark.parametrize("dk,dv,rot,pairs", [(128, 128, 128, False), (64, 64, 32, False), (128, 64, 64, True), (96, 72, 96, False),
                                             (64, 64, 12, True), (64, 64, 0, False), (16, 8, 16, False), (512, 64, 64, False)])
@pytest.mark.parametrize("norm", ["none", "whole", "unit", "shared"])
@pytest.mark.parametrize("n,kv", [(1, 2), (597, 1), (7, 0)])
def test_prepare_by_pieces_is_the_general_kernel(dk, dv, rot, pairs, norm, n, kv):
    """Both kernels compute in float32 and round once: each is within one bfloat16 rounding (2^-9 of the number, and float32's
    error beside it) of the definition in float64, they differ by two at most, and values are copied."""
    from llm_rs_b200 import ops
    torch.manual_seed(dk + rot + n)
    heads, page = 4, 16
    kvh = max(kv, 1)
    q0 = torch.randn(n, heads * dk + 8, device=DEV).bfloat16()
    k = torch.randn(n, kvh * dk + 16, device=DEV).bfloat16()[:, : kvh * dk] if kv else None
    v = torch.randn(n, kvh * dv, device=DEV).bfloat16() if kv else None
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    n_pages = -(-(n + 5) // page)
    table = torch.randperm(n_pages, device=DEV).to(torch.int32).view(1, n_pages)
    ctx = SimpleNamespace(positions=i32(list(range(5, n + 5))), token_req=i32([0] * n))
    inv_freq = 10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64, device=DEV) / max(rot // 2, 1))
    wq = wk = None
    if norm in ("whole", "shared"):
        wq = torch.rand(dk if norm == "shared" else heads * dk, device=DEV) + 0.5
        wk = torch.rand(dk if norm == "shared" else kvh * dk, device=DEV) + 0.5
    got = []
    for generic in (True, False):
        q = q0.clone()[:, : heads * dk]
        cache = torch.zeros(n_pages, kvh, page * (dk + dv), device=DEV).bfloat16()
        ops.scored_generic_only(generic)
        try:
            ops.scored_prepare(q, k, v, wq, wk, inv_freq, ctx, table, cache if kv else None, heads, kvh, dk, dv, rot, page, 1e-6,
                               unit_heads=norm == "unit", shared_head_norm=norm == "shared", pairs=pairs)
        finally:
            ops.scored_generic_only(False)
        got.append((q.float(), cache.float()))
    for a, b in zip(*got):
        assert bool(((a - b).abs() <= 2.0 ** -7 * a.abs() + 1e-5).all())
    want = lambda x, h, w: _prepared(x, h, dk, norm, w, inv_freq, ctx.positions, rot, pairs)
    close = lambda a, b: bool(((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 1e-5).all())
    want_q = want(q0[:, : heads * dk], heads, wq).flatten(1)
    page_of, slot = table[0, ctx.positions.long() // page].long(), ctx.positions.long() % page
    for q, cache in got:
        assert close(q, want_q)
        if kv:
            keys = cache[:, :, : page * dk].unflatten(2, (page, dk))[page_of, :, slot]
            values = cache[:, :, page * dk:].unflatten(2, (page, dv))[page_of, :, slot]
            assert close(keys, want(k, kvh, wk)) and torch.equal(values.flatten(1), v.float())


def test_prepare_of_rows_of_48_kilobytes():
    """The general kernel's rows fill what a kernel may have without asking, beside a reduction of its own."""
    from llm_rs_b200 import ops
    heads, kv, d, page = 88, 8, 128, 16
    q, k, v = (torch.randn(3, h * d, device=DEV) for h in (heads, kv, kv))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    ctx = SimpleNamespace(positions=i32([0, 1, 2]), token_req=i32([0] * 3))
    cache = torch.zeros(1, kv, page * 2 * d, device=DEV)
    q0 = q.clone()
    ops.scored_prepare(q, k, v, None, None, torch.zeros(0, dtype=torch.float64, device=DEV), ctx, i32([[0]]), cache, heads, kv, d, d, 0,
                       page, 1e-6)
    assert torch.equal(q, q0) and torch.equal(cache[0, :, : 3 * d], k.view(3, kv, d).transpose(0, 1).flatten(1))
