"""Prefill attention beside cells of the cache that hold no key of the request: the rest of its last page, what lies before its
window, pages of nobody. Whatever stands there, infinities and NaN too, every output keeps its bits."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D = 128


def _case(lens, cached, page, window, keep, chunk, kv, seed):
    """The step's arrays, its cache and the cells that no query of the step may see."""
    from llm_rs_b200 import host
    g = torch.Generator().manual_seed(seed)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    per = [-(-(c + n) // page) for n, c in zip(lens, cached)]
    order = torch.randperm(sum(per) + 2, generator=g).tolist()
    table = torch.full((len(lens), max(per)), order[-1], dtype=torch.int32)
    cache = torch.randn(sum(per) + 2, kv, 2, page, D, generator=g).to(torch.bfloat16)
    foreign = torch.ones(sum(per) + 2, page, dtype=torch.bool)
    at = 0
    for r, (n, c) in enumerate(zip(lens, cached)):
        pages = order[at:at + per[r]]
        at += per[r]
        table[r, :per[r]] = torch.tensor(pages, dtype=torch.int32)
        floor = c // chunk * chunk if chunk else (max(0, c - window + 1) if window else 0)
        for key in range(c + n):
            if key >= floor or key < keep:
                foreign[pages[key // page], key % page] = False
    tiles, _, _, _ = host.plan_paged_attention(np.array(lens, np.int32), np.array(cached, np.int32), 64)
    ctx = SimpleNamespace(q_start=i32([sum(lens[:r]) for r in range(len(lens))]), n_new=i32(lens), cached_len=i32(cached))
    return ctx, torch.from_numpy(tiles.copy()).to(DEV), table.to(DEV), cache.to(DEV), foreign.to(DEV), g


@pytest.mark.parametrize("tc", [1, 2, 0])
@pytest.mark.parametrize("page", [16, 48, 64])
@pytest.mark.parametrize("lens,cached", [([20], [500]), ([8, 3, 64], [0, 77, 2000]), ([200, 129, 5], [45, 128, 127]), ([128, 16], [128, 112])])
@pytest.mark.parametrize("window,keep,chunk", [(0, 0, 0), (257, 0, 0), (100, 5, 0), (20, 40, 0), (64, 16, 0), (0, 0, 100)])
def test_cells_that_no_query_sees(tc, page, lens, cached, window, keep, chunk):
    from llm_rs_b200 import ops
    heads, kv = 4, 2
    ctx, tiles, table, cache, foreign, g = _case(lens, cached, page, window, keep, chunk, kv, sum(lens) + page + window)
    q = torch.randn(sum(lens), heads * D, generator=g).to(DEV, torch.bfloat16)
    where = foreign[:, None, None, :, None]
    outs = []
    for fill in (0.0, float("inf"), float("nan")):
        c = torch.where(where, torch.tensor(fill, device=DEV, dtype=torch.bfloat16), cache).contiguous()
        for scored in (True,) if keep or chunk else (True, False):
            out = torch.full_like(q, 7.0)
            if scored:
                mask = ops.MASK_CHUNK if chunk else (ops.MASK_WINDOW if window else ops.MASK_CAUSAL)
                ops.scored_prefill(q, out, c.view(c.size(0), kv, -1), tiles, tiles.size(0), ctx, table, heads, kv, D, D, page, 0.09,
                                   20.0, None, mask, chunk or window, prefer_tc=tc, keep=keep)
            else:
                ops.attn_prefill(q, out, c.view(c.size(0), kv, -1), tiles, tiles.size(0), ctx.q_start, ctx.n_new, ctx.cached_len, table,
                                 heads, kv, D, page, window, 0.09, prefer_tc=tc)
            outs.append((fill, scored, out))
    ops.check_attention_error()
    for fill, scored, out in outs:
        assert torch.isfinite(out).all(), (fill, scored)
        assert torch.equal(out, next(o for f, s, o in outs if f == 0.0 and s == scored)), (fill, scored)


@pytest.mark.parametrize("tc", [2, 0])
@pytest.mark.parametrize("scored", [False, True])
@pytest.mark.parametrize("page,window", [(16, 0), (64, 90)])
def test_later_blocks_of_a_short_portion(tc, scored, page, window):
    """A portion of more than 64 tokens beside short ones: the first 64 queries keep their bits whatever the tokens behind them hold,
    as they do on mma.sync, and the two kernels agree to bfloat16's rounding."""
    from llm_rs_b200 import ops
    heads, kv, lens, cached = 4, 2, [100, 2, 2, 127, 3], [500, 500, 30, 61, 500]
    ctx, tiles, table, cache, _, g = _case(lens, cached, page, window, 0, 0, kv, 5)
    q = torch.randn(sum(lens), heads * D, generator=g).to(DEV, torch.bfloat16)

    def run(c, how):
        out = torch.full_like(q, 7.0)
        if scored:
            ops.scored_prefill(q, out, c.view(c.size(0), kv, -1), tiles, tiles.size(0), ctx, table, heads, kv, D, D, page, 0.09, 20.0, None,
                               ops.MASK_WINDOW if window else ops.MASK_CAUSAL, window, prefer_tc=how)
        else:
            ops.attn_prefill(q, out, c.view(c.size(0), kv, -1), tiles, tiles.size(0), ctx.q_start, ctx.n_new, ctx.cached_len, table,
                             heads, kv, D, page, window, 0.09, prefer_tc=how)
        return out

    want = run(cache, tc)
    other = run(cache, 2 - tc)
    assert (want - other).abs().max().item() <= 0.03 * other.abs().max().item()
    bad = cache.clone()
    for r, at in ((0, 64), (3, 120)):
        key = cached[r] + at
        bad[int(table[r, key // page]), :, :, key % page] = float("nan")
    got = run(bad, tc)
    ops.check_attention_error()
    for r in range(len(lens)):
        first = sum(lens[:r])
        n = min(lens[r], 64) if r in (0, 3) else lens[r]
        assert torch.isfinite(want[first: first + n]).all()
        assert torch.equal(got[first: first + n], want[first: first + n]), r
