"""Long prompt portions through latent attention with keys and values made for the step (parts/latent_attention.py, the tcgen05
kernel with latent keys) against the folded form over the pages and against a plain float64 evaluation: own keys of 64 and 128
channels, shared parts of 16 to 64, windows that end inside a tile and none, portions on top of cached keys, short portions
and single tokens in the same step, with and without the gate. Both forms round queries, keys, values or latents to bfloat16
once each: an element may be off by some 2^-7 of the largest output."""
import math
import sys
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 16


class _Ctx(SimpleNamespace):
    def plan(self, key):
        return self.plans[key]

    def scratch(self, name, n_floats):
        return torch.zeros((max(n_floats, 1),), dtype=torch.float32, device=DEV)


def _step(part, n_new, cached):
    from llm_rs_b200.parts.base import StepInfo
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    a32 = lambda v: np.asarray(v, np.int32)
    q_start = [sum(n_new[:r]) for r in range(len(n_new))]
    slots = list(range(len(n_new)))
    plan = part.plan(StepInfo(sum(n_new), len(n_new), a32(q_start), a32(n_new), a32(cached), a32(slots), [], [], PAGE, False))
    view = SimpleNamespace(arrays={k: torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for k, v in plan.arrays.items()},
                           values=plan.values)
    return _Ctx(n_tokens=sum(n_new), n_requests=len(n_new), q_start=i32(q_start), n_new=i32(n_new), cached_len=i32(cached),
                slot_ids=i32(slots), token_req=i32([r for r, n in enumerate(n_new) for _ in range(n)]),
                positions=i32([c + i for c, n in zip(cached, n_new) for i in range(n)]), plans={part.plan_key(): view})


def _plain(part, w, x, dn, dr, rank, nh, window, cached, latents, parts):
    """One request's outputs in float64 from all its latents and rotated parts (its new ones last)."""
    n = x.size(0)
    q = (x @ w["q"].t()).view(n, nh, dn + dr)
    pos = torch.arange(cached, cached + n, dtype=torch.float64)[:, None]
    f = 900.0 ** (-2.0 * torch.arange(dr // 2, dtype=torch.float64) / dr)
    rot = lambda t, c, s: torch.cat([t[..., : dr // 2] * c - t[..., dr // 2:] * s, t[..., : dr // 2] * s + t[..., dr // 2:] * c], -1)
    c, s = (pos * f).cos(), (pos * f).sin()
    q_rot = rot(q[:, :, dn:], c[:, None], s[:, None])
    dkv = x @ w["dkv"].t()
    new = dkv[:, :rank] / torch.sqrt((dkv[:, :rank] ** 2).mean(-1, keepdim=True) + 1e-6) * w["dkv.norm"]
    latents, parts = torch.cat([latents, new]), torch.cat([parts, rot(dkv[:, rank:], c, s)])
    key = torch.arange(cached + n)[None]
    see = (key <= pos) & ((key > pos - window) if window else torch.tensor(True))
    out = torch.empty(n, nh, 128, dtype=torch.float64)
    for h in range(nh):
        k, v = latents @ w["uk"].view(nh, dn, rank)[h].t(), latents @ w["uv"].view(nh, 128, rank)[h].t()
        score = (q[:, h, :dn] @ k.t() + q_rot[:, h] @ parts.t()) * part.scale
        out[:, h] = torch.softmax(score.masked_fill(~see, -math.inf), dim=1) @ v
    if "g" in w:
        out = out * torch.sigmoid(x @ w["g"].t())[..., None]
    return out.reshape(n, -1) @ w["o"].t(), latents, parts


def _small_part(window):
    """A part of 8 heads of 64 + 32 over latents of 128, bound to random weights."""
    from llm_rs_b200.parts import Runtime
    from llm_rs_b200.parts import latent_attention as L
    g = torch.Generator().manual_seed(5)
    part = L.LatentAttention(96, 8, 64, 32, 128, 128, 96 ** -0.5, 900.0, window=window, prefix="m.")
    part.bind({s.name: (torch.ones(s.shape) if len(s.shape) == 1 else torch.randn(s.shape, generator=g) * s.shape[1] ** -0.5)
               .to(DEV, torch.float32 if len(s.shape) == 1 else torch.bfloat16) for s in part.weight_specs()},
              Runtime(torch.device(DEV), torch.bfloat16, 4096))
    return part


def _small_cache(n_requests, n_pages):
    pages = torch.zeros((n_requests * n_pages, 1, PAGE * (128 + 32)), dtype=torch.bfloat16, device=DEV)
    planes = [pages[:, :, : PAGE * 128].unflatten(2, (PAGE, 128)), pages[:, :, PAGE * 128:].unflatten(2, (PAGE, 32))]
    table = torch.arange(n_requests * n_pages, dtype=torch.int32, device=DEV).view(n_requests, n_pages)
    return SimpleNamespace(planes=planes, block_table=table, page_size=PAGE, owns=True, state={})


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("lens", [(64, 70), (130, 64), (128, 81), (200, 255)])
def test_a_neighbours_numbers_do_not_reach_a_request(lens, bad):
    """Both requests' keys are made for the step: what the second one holds must not change a bit of the first one's output."""
    part = _small_part(window=0)
    x = torch.randn(sum(lens), 96, generator=torch.Generator().manual_seed(1)).to(DEV, torch.bfloat16)
    ctx = _step(part, lens, (0, 0))
    assert ctx.plans[part.plan_key()].values["n_long"] == sum(-(-n // 128) for n in lens)
    want = part.forward(x, ctx, _small_cache(2, 16))
    x = x.clone()
    x[lens[0]:] = bad
    got = part.forward(x, ctx, _small_cache(2, 16))
    assert torch.equal(got[: lens[0]], want[: lens[0]])
    assert torch.isnan(got[lens[0]:]).all()


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("window,n,cached,at", [(0, 100, 0, 99), (0, 200, 60, 131), (0, 130, 0, 64), (20, 150, 40, 30),
                                                (20, 100, 40, 38), (50, 260, 0, 128)])
def test_a_key_that_is_not_finite_reaches_its_queries_only(window, n, cached, at, bad):
    """The latent at position ``at`` (a cached one, or a new one) is ``bad`` in one channel: the queries before it, and those
    whose window has passed it, keep every bit."""
    part = _small_part(window)
    x = torch.randn(n, 96, generator=torch.Generator().manual_seed(2)).to(DEV, torch.bfloat16)
    ctx = _step(part, (n,), (cached,))
    assert ctx.plans[part.plan_key()].values["n_long"] == -(-n // 128)

    def run(poison):
        cache = _small_cache(1, 20)
        cache.planes[0].copy_(torch.randn(cache.planes[0].shape, generator=torch.Generator().manual_seed(3)))
        if poison and at < cached:
            cache.planes[0][at // PAGE, 0, at % PAGE, 77] = bad
        rows = x.clone()
        if poison and at >= cached:
            rows[at - cached] = bad
        return part.forward(rows, ctx, cache)
    want, got = run(False), run(True)
    pos = cached + torch.arange(n, device=DEV)
    sees = (pos >= at) & ((pos < at + window) if window else True)
    assert torch.isfinite(want).all() and sees.any() and not sees.all()
    assert torch.equal(got[~sees], want[~sees])
    assert torch.isnan(got[sees]).all()


@pytest.mark.parametrize("dn,dr,rank,nh,window,gated,cuts", [
    (128, 64, 512, 8, 0, True, [(300, 64), (129, 1), (70, 200)]), (64, 32, 128, 8, 100, True, [(128, 90), (257, 64), (64, 13)]),
    (128, 16, 64, 5, 257, False, [(65, 700), (200, 127)]), (64, 64, 256, 16, 1024, True, [(1200, 1), (333, 1)]),
    (128, 48, 192, 8, 1, True, [(130, 66), (64, 64)]), (128, 64, 512, 16, 128, True, [(255, 256, 1, 40, 64)])])
def test_long_portions_with_keys_made_for_the_step(dn, dr, rank, nh, window, gated, cuts, monkeypatch):
    from llm_rs_b200.parts import Runtime
    from llm_rs_b200.parts import latent_attention as L
    monkeypatch.setattr(L, "EXPAND_BESIDE", 0)      # also beside other tokens, and over few keys
    monkeypatch.setattr(L, "EXPAND_MIN_KEYS", 0)
    g = torch.Generator().manual_seed(dn + dr + nh)
    D = 96
    part = L.LatentAttention(D, nh, dn, dr, 128, rank, (dn + dr) ** -0.5, 900.0, window=window, gated=gated, prefix="m.")
    w = {s.name[2:]: ((1.0 + 0.1 * torch.randn(s.shape, generator=g)) if len(s.shape) == 1 else
                      torch.randn(s.shape, generator=g) * s.shape[1] ** -0.5).bfloat16().float() for s in part.weight_specs()}
    part.bind({"m." + k: v.to(DEV, torch.float32 if v.dim() == 1 else torch.bfloat16) for k, v in w.items()},
              Runtime(torch.device(DEV), torch.bfloat16, 4096))
    wd = {k: v.double() for k, v in w.items()}
    R = len(cuts[0])
    total = [sum(c[r] for c in cuts) for r in range(R)]
    width = -(-max(total) // PAGE)
    table = torch.randperm(R * width, generator=g).to(torch.int32).view(R, width).to(DEV)
    pages = torch.zeros((R * width, 1, PAGE * (rank + dr)), dtype=torch.bfloat16, device=DEV)
    planes = [pages[:, :, : PAGE * rank].unflatten(2, (PAGE, rank)), pages[:, :, PAGE * rank:].unflatten(2, (PAGE, dr))]
    cache = SimpleNamespace(planes=planes, block_table=table, page_size=PAGE, owns=True, state={})
    at = [0] * R
    kept = [(torch.zeros(0, rank, dtype=torch.float64), torch.zeros(0, dr, dtype=torch.float64)) for _ in range(R)]
    for cut in cuts:
        cut = list(cut)
        x = torch.randn(sum(cut), D, generator=g).bfloat16()
        ctx = _step(part, cut, at)
        assert ctx.plans[part.plan_key()].values["n_long"] == sum(-(-n // 128) for n in cut if n >= L.EXPAND_MIN_TOKENS)
        got = part.forward(x.to(DEV), ctx, cache).float().cpu()
        L.EXPAND_MIN_TOKENS, saved = 1 << 30, L.EXPAND_MIN_TOKENS
        try:
            folded_ctx = _step(part, cut, at)
        finally:
            L.EXPAND_MIN_TOKENS = saved
        folded = part.forward(x.to(DEV), folded_ctx, cache).float().cpu()
        o = 0
        for r, n in enumerate(cut):
            want, *kept[r] = _plain(part, wd, x[o:o + n].double(), dn, dr, rank, nh, window, at[r], *kept[r])
            scale = float(want.abs().max())
            assert float((got[o:o + n].double() - want).abs().max()) <= 0.03 * scale, (cut, r)
            assert float((got[o:o + n] - folded[o:o + n]).abs().max()) <= 0.03 * scale, (cut, r)
            o += n
            at[r] += n
        if window:      # pages that no later query may see are given back: nobody may read them
            for r in range(R):
                for pg in range(max(0, at[r] - window + 1) // PAGE):
                    if int(table[r, pg]) >= 0:
                        pages[int(table[r, pg])] = float("nan")
                        table[r, pg] = -1


@pytest.mark.parametrize("page", [16, 8])
def test_single_tokens_between_long_portions(page, monkeypatch):
    """The folded form takes the tokens between long portions alone (pages of 8 keys: by the kernel of few tokens); the same
    numbers as from the folded form for all."""
    from llm_rs_b200.parts import latent_attention as L
    monkeypatch.setattr(sys.modules[__name__], "PAGE", page)
    monkeypatch.setattr(L, "FOLD_GAP", 50)
    part = _small_part(window=0)
    n_new, cached = (1, 3, 140, 1, 40, 2, 200, 1), (30, 0, 5, 100, 30, 64, 0, 7)
    x = torch.randn(sum(n_new), 96, generator=torch.Generator().manual_seed(6)).to(DEV, torch.bfloat16)
    fill = torch.randn((8 * 256 // page, 1, page * 160), generator=torch.Generator().manual_seed(7)).to(DEV, torch.bfloat16)

    def run():
        ctx = _step(part, n_new, cached)
        cache = _small_cache(8, 256 // page)
        for plane, width, at in ((cache.planes[0], 128, 0), (cache.planes[1], 32, page * 128)):
            plane.copy_(fill[:, :, at: at + page * width].unflatten(2, (page, width)))
        return ctx.plans[part.plan_key()].values, part.forward(x, ctx, cache).float()
    values, got = run()
    assert values["n_long"] == 2 + 1 + 2 and values["others"] == ((0, 4), (144, 187), (387, 388))
    monkeypatch.setattr(L, "EXPAND_MIN_TOKENS", 1 << 30)
    values, want = run()
    assert values["n_long"] == 0
    assert float((got - want).abs().max()) <= 0.03 * float(want.abs().max())
