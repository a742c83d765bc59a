"""Latent attention: all heads share one cached row per token."""
from __future__ import annotations

import math
import os
from types import SimpleNamespace
from typing import Mapping, Optional

import numpy as np
import torch

from .. import ops
from .base import Mixer, Plan, Runtime, StepInfo
from .linear import Linear
from .registry import register
from .spec import CacheNeed, WeightSpec


# Prompt portions in bfloat16 take the tensor-core kernel from this many tokens a step on; LLMRS_LATENT_MMA=0 keeps the
# CUDA-core kernel for everything.
_LATENT_MMA = os.environ.get("LLMRS_LATENT_MMA", "1") != "0"
PREFILL_MIN_TOKENS = 32
# Portions of at least EXPAND_MIN_TOKENS tokens that see at most EXPAND_MAX_KEYS keys per token of theirs have the keys and
# values of what they see made for the step and take the tcgen05 attention kernel: the folded form needs no keys or values but
# 3.4 times the multiplications (a latent of 512 against heads of 192 and 128) and walks a tile's keys on mma.sync. Measured,
# 16 heads, a whole mixer, folded against made (us): 2,000 tokens through a window of 1,024 799 / 133; 64 tokens after 4,096
# 793 / 119, after 8,000 1,486 / 187; 32 after 2,048 418 / 77, after 256 98 / 55. Fewer tokens over more keys were not
# measured and stay folded.
# A step with other tokens runs the folded kernel all the same, which takes a few tokens more along for little: there the long
# portions need EXPAND_BESIDE tokens together. Single tokens after 900 keys + a portion after 800, folded together / the portion
# apart (us): 1 + 64 197 / 216, 63 + 64 240 / 282, 1 + 128 205 / 225, 1 + 256 228 / 238, 8 + 256 276 / 242, 1 + 512 284 / 253,
# 63 + 512 502 / 312.
# A portion over fewer than EXPAND_MIN_KEYS keys is folded at no more cost: heads of 64 + 32, a latent of 256, 40 tokens after none
# 45 / 49, 64 after none 50 / 50, 32 after 256 82 / 51; heads of 128 + 64, a latent of 512, 32 after none 50 / 50.
EXPAND_MIN_TOKENS, EXPAND_MIN_KEYS, EXPAND_MAX_KEYS, EXPAND_BESIDE = 32, 64, 128, 320
EXPAND_ALIGN = 128      # keys per tile of that kernel
# Tokens of long portions between two runs of other tokens that the folded form's products take along: fewer cost less than
# another launch of each of the two products.
FOLD_GAP = 256


def rescaled_frequencies(dims: int, base: float, scaling: Optional[Mapping] = None):
    """(inverse frequencies float64 [dims/2], magnitude) of a rotation of ``dims`` entries: ``f_i = base^(-2i/dims)``.

    ``scaling`` (factor, original, fast, slow) stretches the slow pairs for contexts longer than the ``original`` one
    (YaRN: Peng, Quesnelle, Fan, Shippole, "YaRN: Efficient Context Window Extension of Large Language Models"). A
    pair that turns ``t`` times within the original context has index ``d(t) = dims * ln(original / (2 pi t)) / (2 ln
    base)``; pairs below ``lo = max(floor(d(fast)), 0)`` keep their frequency, pairs above ``hi = min(ceil(d(slow)),
    dims - 1)`` have it divided by ``factor``, and between them the two are blended by ``ramp_i = clamp((i - lo) /
    max(hi - lo, 0.001), 0, 1)``: ``f_i / factor * ramp_i + f_i * (1 - ramp_i)``. Cosines and sines are multiplied by
    the magnitude ``0.1 ln(factor) + 1``."""
    i = torch.arange(dims // 2, dtype=torch.float64)
    f = float(base) ** (-2.0 * i / max(dims, 1))
    if not scaling:
        return f, 1.0
    factor, original = float(scaling["factor"]), float(scaling["original"])
    index = lambda turns: dims * math.log(original / (2.0 * math.pi * turns)) / (2.0 * math.log(float(base)))
    lo = max(math.floor(index(float(scaling["fast"]))), 0)
    hi = min(math.ceil(index(float(scaling["slow"]))), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / factor * ramp + f * (1.0 - ramp), 0.1 * math.log(factor) + 1.0


def portion_tiles(q_start, n_new, tile_tokens: int) -> np.ndarray:
    """int32 [n, 2]: (first token of the step, tokens) of tiles of at most ``tile_tokens`` consecutive tokens that do
    not cross a request."""
    firsts, counts = [], []
    for qs, n in zip(np.asarray(q_start).tolist(), np.asarray(n_new).tolist()):
        a = np.arange(0, n, tile_tokens, dtype=np.int32)
        firsts.append(qs + a)
        counts.append(np.minimum(tile_tokens, n - a))
    if not firsts:
        return np.zeros((0, 2), np.int32)
    return np.stack([np.concatenate(firsts), np.concatenate(counts)], axis=1).astype(np.int32)


def other_ranges(q_start, n_new, is_long, n_tokens: int):
    """The step's tokens that are of no long portion, as ranges (first, end); ranges less than FOLD_GAP apart are one."""
    ranges, at = [], 0
    for r in np.nonzero(is_long)[0].tolist() + [None]:
        end = n_tokens if r is None else int(q_start[r])
        if end > at:
            if ranges and at - ranges[-1][1] <= FOLD_GAP:
                ranges[-1] = (ranges[-1][0], end)
            else:
                ranges.append((at, end))
        at = end if r is None else end + int(n_new[r])
    return tuple(ranges)


def expanded_rows(n_new, cached, window: int, row_bytes: int):
    """Per request the position of the first key that is made for the step (a multiple of EXPAND_ALIGN), how many rows are made
    for it, and whether the request's portion is taken that way (``row_bytes`` a row; 0: none are; at most
    ``ops.LATENT_EXPAND_BYTES`` together). A request's rows are whole tiles of the attention kernel, zeros past its last key:
    a tile that ran on into the next request's rows would multiply their values by weights of zero, which is no number where
    they are infinite."""
    lo = np.maximum(0, cached - window + 1) if window > 0 else np.zeros_like(cached)
    first = lo // EXPAND_ALIGN * EXPAND_ALIGN
    keys = cached + n_new - first
    counts = -(-keys // EXPAND_ALIGN) * EXPAND_ALIGN
    is_long = (n_new >= EXPAND_MIN_TOKENS) & (keys >= EXPAND_MIN_KEYS) & (keys <= EXPAND_MAX_KEYS * n_new) & (row_bytes > 0)
    room = ops.LATENT_EXPAND_BYTES
    for r in np.nonzero(is_long)[0].tolist():      # one that does not fit leaves the room to those behind it
        need = int(counts[r]) * row_bytes
        is_long[r] = need <= room
        room -= need if need <= room else 0
    if ((n_new > 0) & ~is_long).any() and int(n_new[is_long].sum()) < EXPAND_BESIDE:
        is_long[:] = False
    return first, np.where(is_long, counts, 0), is_long


class _TokenRange:
    """Tokens a .. b - 1 of a step, as the attention of few tokens reads them."""

    def __init__(self, ctx, a: int, b: int):
        self.positions, self.token_req = ctx.positions[a:b], ctx.token_req[a:b]
        if hasattr(ctx, "scratch"):
            self.scratch = ctx.scratch


@register("mixer", "latent_attention")
class LatentAttention(Mixer):
    """Attention whose keys and values are up-projections of a small cached latent.

    Per token the down-projection gives ``rank + rot_dim`` numbers: the first ``rank``, RMS-normed with a plain
    weight, are the latent c; the last ``rot_dim`` (rotated by position, not normed) are a key part shared by all
    heads. Only these are cached. A query head is [``dim`` unrotated | ``rot_dim`` rotated]; head h's unrotated key
    is ``W_uk,h c`` and its value ``W_uv,h c``. The score is ``(q_n . k_n + q_r . k_r) * scale`` over the causal keys
    (the last ``window`` of them when ``window`` > 0), ordinary softmax; head h's output is multiplied by
    ``sigmoid(W_g x)_h`` when ``gated``; then the output projection.

    Computed in the folded form: ``qa_h = W_uk,h^T q_n,h`` (a batched product), attention over the cached rows with
    values c, then ``W_uv,h`` on the result (a batched product): the cache is read once for all heads and no key or
    value is ever materialised. The rotation pairs entry i of the rotated part with entry i + rot_dims/2 for the first
    ``rot_dims`` entries (``rot_pairing`` "half"), or entry 2i with 2i + 1 ("neighbours"), angle ``position *
    rot_base^(-2i/rot_dims)``; ``rot_scaling`` rescales the frequencies (``rescaled_frequencies``).

    ``q_rank`` > 0: the queries go through a latent of their own, ``q = W_uq rmsnorm(W_dq x)`` with a plain norm
    weight; the down-projection shares the product of the gates and the key/value down-projection.

    A layer with ``shares_cache`` has no down-projection: its run-order entry reads another entry's pages
    (``RunStep.cache_of``) with its own up-projections, queries and window. ``cache_window`` is the window the pages
    are kept for (the widest window of the layers that read them; default: this layer's).

    ``names`` maps the roles q, dq, dq_norm, uq, dkv, dkv_norm, uk, uv, g, o to tensor names after the prefix.
    """
    ROLES = ("q", "dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "g", "o")
    PAIRINGS = ("half", "neighbours")

    def __init__(self, hidden_size: int, n_heads: int, dim: int, rot_dim: int, vdim: int, rank: int, scale: float,
                 rot_base: float, rot_dims: Optional[int] = None, window: int = 0, cache_window: Optional[int] = None,
                 norm_eps: float = 1e-6, gated: bool = True, shares_cache: bool = False, q_rank: int = 0,
                 rot_pairing: str = "half", rot_scaling: Optional[Mapping] = None, names=None, prefix: str = ""):
        self.hidden_size, self.n_heads, self.dim, self.rot_dim, self.vdim = hidden_size, n_heads, dim, rot_dim, vdim
        self.rank, self.scale, self.rot_base = rank, float(scale), float(rot_base)
        self.rot_dims = rot_dim if rot_dims is None else int(rot_dims)
        if self.rot_dims % 2 or not 0 <= self.rot_dims <= rot_dim:
            raise ValueError(f"{self.rot_dims} rotated dimensions of a rotated part of {rot_dim}")
        if rot_pairing not in self.PAIRINGS:
            raise ValueError(f"unknown rot_pairing {rot_pairing!r}; known: {self.PAIRINGS}")
        self.q_rank, self.rot_pairing = int(q_rank), rot_pairing
        self.rot_scaling = dict(rot_scaling) if rot_scaling else None
        if rank > 512:
            raise ValueError(f"a latent of {rank}: the attention kernel takes at most 512")
        self.window = int(window)
        self.cache_window = self.window if cache_window is None else int(cache_window)
        if self.cache_window and (self.window == 0 or self.window > self.cache_window):
            raise ValueError(f"pages kept for the last {self.cache_window} keys cannot serve a window of "
                             f"{self.window or 'all'} keys")
        self.norm_eps, self.gated, self.shares_cache = float(norm_eps), bool(gated), bool(shares_cache)
        self.prefix = prefix
        self.names = {"q": "q", "dq": "dq", "dq_norm": "dq.norm", "uq": "uq", "dkv": "dkv", "dkv_norm": "dkv.norm",
                      "uk": "uk", "uv": "uv", "g": "g", "o": "o"}
        self.names.update(names or {})
        if set(self.names) != set(self.ROLES):
            raise ValueError(f"names may rename {self.ROLES}, got {sorted(set(self.names) - set(self.ROLES))}")
        self.q_width = n_heads * (dim + rot_dim)
        self._tile = None

    def _name(self, role: str) -> str:
        return self.prefix + self.names[role]

    def weight_specs(self):
        H, nh, nm = self.hidden_size, self.n_heads, self._name
        specs = [WeightSpec(nm("uk"), (nh * self.dim, self.rank)),
                 WeightSpec(nm("uv"), (nh * self.vdim, self.rank)), WeightSpec(nm("o"), (H, nh * self.vdim))]
        if self.q_rank:
            specs += [WeightSpec(nm("dq"), (self.q_rank, H)), WeightSpec(nm("dq_norm"), (self.q_rank,), role="norm"),
                      WeightSpec(nm("uq"), (self.q_width, self.q_rank))]
        else:
            specs.append(WeightSpec(nm("q"), (self.q_width, H)))
        if self.gated:
            specs.append(WeightSpec(nm("g"), (nh, H)))
        if not self.shares_cache:
            specs += [WeightSpec(nm("dkv"), (self.rank + self.rot_dim, H)),
                      WeightSpec(nm("dkv_norm"), (self.rank,), role="norm")]
        return specs

    def bind(self, tensors, runtime: Runtime):
        nm, nh = self._name, self.n_heads
        self.act_dtype = runtime.act_dtype
        ws = [tensors[nm("dq") if self.q_rank else nm("q")]]
        self.q_up = self.q_norm_w = None
        if self.q_rank:
            self.q_up = Linear(tensors[nm("uq")], None, runtime.act_dtype)
            self.q_norm_w = tensors[nm("dq_norm")].to(torch.float32).contiguous()
        if self.gated:
            ws.append(tensors[nm("g")])
        if not self.shares_cache:
            ws.append(tensors[nm("dkv")])
        dt = ws[0].dtype if all(w.dtype == ws[0].dtype for w in ws) else torch.float32
        # One product for the queries, the gates and the down-projection: they read the same input.
        self.in_proj = Linear(torch.cat([w.to(dt) for w in ws], dim=0).contiguous(), None, runtime.act_dtype)
        self.o_proj = Linear(tensors[nm("o")], None, runtime.act_dtype)
        # W_uk,h transposed to [rank, dim]: the folded query is an ordinary product with it.
        self.w_uk_t = tensors[nm("uk")].view(nh, self.dim, self.rank).transpose(1, 2).contiguous()
        self.w_uv = tensors[nm("uv")].view(nh, self.vdim, self.rank).contiguous()
        # For portions whose keys and values are made for the step: both up-projections as one product's weight.
        self.w_expand = None
        q_row = self.q_width if self.q_rank else self.in_proj.weight.size(0)      # the kernel reads rows of q 16 bytes at a time
        if (q_row % 8 == 0 and runtime.act_dtype == torch.bfloat16 and self.w_uv.dtype == self.w_uk_t.dtype == torch.bfloat16 and self.dim in (64, 128)
                and self.vdim == 128 and self.rank % 64 == 0 and self.rot_dim % 16 == 0 and 0 < self.rot_dim <= 64):
            self.w_expand = torch.cat([tensors[nm("uk")], tensors[nm("uv")]], dim=0).contiguous()
        self.latent_norm_w = None if self.shares_cache else tensors[nm("dkv_norm")].to(torch.float32).contiguous()
        self.open_gate = torch.full((1, nh), 30.0, dtype=runtime.act_dtype, device=runtime.device)
        inv_freq, self.rot_magnitude = rescaled_frequencies(self.rot_dims, self.rot_base, self.rot_scaling)
        self.inv_freq = inv_freq.to(runtime.device)

    def cache_need(self):
        if self.shares_cache:
            return None
        return CacheNeed("window" if self.cache_window > 0 else "full", 1, self.rank, self.cache_window,
                         planes=(self.rank, self.rot_dim))

    # -- the step's plan: tiles of a prompt's tokens for the tensor-core kernel -------------------------------------
    def _tile_tokens(self) -> int:
        if self._tile is None:      # asked of the kernel library at first use: constructing a part needs no library
            self._tile = ops.latent_prefill_tile_tokens(self.n_heads)
        return self._tile

    def _expand_row_bytes(self) -> int:
        """Bytes of workspace that a visible key takes when its keys and values are made for the step (0: never)."""
        if not _LATENT_MMA or self.w_expand is None:
            return 0
        return 2 * (self.n_heads * (self.dim + self.vdim) + self.rank + self.rot_dim)

    def plan_key(self):
        return ("latent_attention_tiles", self._tile_tokens(), self.window, self._expand_row_bytes())

    def plan(self, step: StepInfo) -> Plan:
        """Steps that bring a prompt's portion are cut into tiles of tokens (none for steps of single tokens, which
        the CUDA-core kernel takes with its keys cut over blocks, and which may be replayed from a graph): long portions
        into tiles of 128 queries over rows that are made for the step (``rows``: a request's first row and the position of
        its first key), the others into the tiles of the kernel that reads the pages."""
        none = np.zeros((0, 2), np.int32)
        if step.for_graph or step.n_tokens < PREFILL_MIN_TOKENS or int(np.max(step.n_new, initial=0)) <= 1:
            return Plan(arrays={"tiles": none, "long": none, "rows": none},
                        values={"n_tiles": 0, "n_long": 0, "n_rows": 0, "others": ((0, step.n_tokens),)})
        n_new, cached = np.asarray(step.n_new, np.int64), np.asarray(step.cached_len, np.int64)
        first, counts, is_long = expanded_rows(n_new, cached, self.window, self._expand_row_bytes())
        tiles = portion_tiles(step.q_start, np.where(is_long, 0, n_new), self._tile_tokens())
        long_tiles = [(r, a) for r in np.nonzero(is_long)[0].tolist() for a in range(0, int(n_new[r]), EXPAND_ALIGN)]
        rows = np.stack([np.cumsum(counts) - counts, first], axis=1).astype(np.int32)
        return Plan(arrays={"tiles": tiles, "long": np.asarray(long_tiles, np.int32).reshape(-1, 2), "rows": rows},
                    values={"n_tiles": int(tiles.shape[0]), "n_long": len(long_tiles), "n_rows": int(counts.sum()),
                            "others": other_ranges(step.q_start, n_new, is_long, step.n_tokens)})

    def _plan_of(self, ctx):
        """The step's plan; outside the step function (a part alone) it is made here, from the device's arrays."""
        if hasattr(ctx, "plan"):
            return ctx.plan(self.plan_key())
        host = lambda t: t.cpu().numpy()
        plan = self.plan(StepInfo(ctx.n_tokens, ctx.n_requests, host(ctx.q_start), host(ctx.n_new), host(ctx.cached_len),
                                  host(ctx.slot_ids), [], [], 0, False))
        return SimpleNamespace(arrays={k: torch.from_numpy(v).to(ctx.n_new.device) for k, v in plan.arrays.items()},
                               values=plan.values)

    def forward(self, x, ctx, cache):
        nh, dn, dr, rank = self.n_heads, self.dim, self.rot_dim, self.rank
        if cache.owns == self.shares_cache:
            raise RuntimeError("a latent attention layer that shares a cache must run as an entry with cache_of "
                               "(and one that owns its cache must not)")
        T = ctx.n_tokens
        proj = self.in_proj.forward(x)
        if self.q_rank:      # queries through their own latent: norm (float32 statistics), then the up-projection
            q = self.q_up.forward(ops.rmsnorm_rows(proj[:, : self.q_rank], self.q_norm_w, self.norm_eps))
            at = self.q_rank
        else:
            q = proj[:, : self.q_width]
            at = self.q_width
        if self.gated:
            gate = proj[:, at: at + nh]
            at += nh
        else:       # sigmoid(+large) = 1: one constant row, read by every token (row stride 0)
            gate = self.open_gate.expand(T, nh)
        dkv = None if self.shares_cache else proj[:, at: at + rank + dr]
        pages = self._pages(cache)
        ops.latent_prepare(q, dkv, self.latent_norm_w, self.inv_freq, ctx, cache.block_table,
                           None if self.shares_cache else pages, cache.page_size, nh, dn, dr, self.rot_dims, rank,
                           self.norm_eps, neighbours=self.rot_pairing == "neighbours", magnitude=self.rot_magnitude)
        plan = self._plan_of(ctx) if _LATENT_MMA and proj.dtype == torch.bfloat16 else None
        n_tiles, n_long = (plan.values["n_tiles"], plan.values["n_long"]) if plan is not None else (0, 0)
        out = torch.empty((T, nh, self.vdim), dtype=proj.dtype, device=proj.device)
        if n_long == 0 or n_tiles:
            self._folded(q, gate, pages, cache, ctx, plan if n_tiles else None, out)
        if n_long:      # (what the folded form left in rows of theirs between its ranges is overwritten)
            c, kr = ops.latent_gather(pages, cache.block_table, ctx, plan.arrays["rows"], plan.values["n_rows"], rank, dr,
                                      cache.page_size, self.window)
            kv = ops.gemm_bf16(c, self.w_expand)
            ops.latent_attention_tc(q, gate, kv, kr, plan.arrays["rows"], plan.arrays["long"], n_long, ctx,
                                    out.view(T, nh * self.vdim), nh, dn, dr, self.window, self.scale)
        return self.o_proj.forward(out.view(T, nh * self.vdim))

    def _folded(self, q, gate, pages, cache, ctx, plan, out) -> None:
        """The attention-weighted latents through the value up-projection into ``out`` [tokens, heads, vdim], for the tokens
        that are of no long portion (``plan``; all of them without one)."""
        nh, dn, dr, rank = self.n_heads, self.dim, self.rot_dim, self.rank
        T = ctx.n_tokens
        ranges = plan.values["others"] if plan is not None else ((0, T),)
        q3 = q.unflatten(1, (nh, dn + dr))
        qa = torch.empty((T, nh, rank), dtype=q.dtype, device=q.device)
        lat = torch.empty((T, nh, rank), dtype=q.dtype, device=q.device)
        for a, b in ranges:
            ops.gemm_batched(q3[a:b, :, :dn], self.w_uk_t, qa[a:b])
        if plan is None or not ops.latent_attention_prefill(
                qa, q, gate, pages, cache.block_table, ctx, plan.arrays["tiles"], plan.values["n_tiles"], lat, nh, dn, dr, rank,
                cache.page_size, self.window, self.scale):
            # Steps of few tokens cut the visible keys over several blocks. The span is what the step's shape implies (the
            # window, else what the block table can hold), not the requests' lengths: a captured step replays it.
            span = self.window if self.window > 0 else cache.block_table.size(1) * cache.page_size
            for a, b in ranges:
                splits, split_keys = ops.latent_attention_splits(
                    b - a, nh, span, ops.sm_count(q.device),
                    mma=b - a <= ops.LATENT_FEW_TOKENS and ops.latent_decode_takes_mma(q.dtype, rank, dr, cache.page_size))
                ops.latent_attention(qa[a:b], q[a:b], gate[a:b], pages, cache.block_table, _TokenRange(ctx, a, b), lat[a:b], nh, dn,
                                     dr, rank, cache.page_size, self.window, self.scale, splits=splits, split_keys=split_keys)
        for a, b in ranges:
            ops.gemm_batched(lat[a:b], self.w_uv, out[a:b])

    @staticmethod
    def _pages(cache):
        """The entry's pages as one tensor [pages, page_size * (rank + rot_dim)]: plane 0 (the latents) and plane 1
        (the rotated key parts) of a page follow one another."""
        p0 = cache.planes[0]
        return p0.as_strided((p0.size(0), p0.stride(0)), (p0.stride(0), 1), p0.storage_offset())
