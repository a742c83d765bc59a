"""The recurrences with a matrix state walked in chunks of sixteen tokens (csrc/state_chunks.cuh) or in turns of four
(csrc/state_walk.cuh), by their heads, and token by token: the same outputs
and states from either, at the edges of chunks, turns, stages and copies, for many requests in one step, with all of a step's requests
in turns or those from some length on. Both are float32 evaluations of one recurrence, each some 1e-6 from 64 bits in the
2-norm at these sizes; single elements may lie sixteen times that apart."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ctx(n_new, cached):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return SimpleNamespace(
        n_tokens=sum(n_new), n_requests=len(n_new), q_start=i32([sum(n_new[:r]) for r in range(len(n_new))]), n_new=i32(n_new),
        cached_len=i32(cached), slot_ids=i32(list(range(len(n_new)))[::-1]),
        token_req=i32([r for r, n in enumerate(n_new) for _ in range(n)]),
        positions=i32([c + i for c, n in zip(cached, n_new) for i in range(n)]))


def _part(kind, d, dv, taps=3):
    from llm_rs_b200.parts.delta_rule import ChannelDelta, GatedDelta, GeneralDelta
    from llm_rs_b200.parts.recurrent import MatrixMemory, Retention
    from llm_rs_b200.parts.ssd import Mamba2
    D = 40
    return D, {"memory": lambda: MatrixMemory(D, 3, d, dv, gate_cap=9.0, prefix="m."),
               "retention": lambda: Retention(D, 3, d, dv, [0.9, 0.0, 1.0], prefix="m."),
               "mamba": lambda: Mamba2(D, 4, dv, d, 2, 3, norm_parts=1, prefix="m."),
               "gated": lambda: GatedDelta(D, 4, 2, d, dv, taps, prefix="m."),
               "channel": lambda: ChannelDelta(D, 4, 2, d, dv, taps, 8, 8, prefix="m."),
               "general": lambda: GeneralDelta(D, 3, d, 8, prefix="m."),
               "mamba of one group": lambda: Mamba2(D, 7, dv, d, 1, 3, norm_parts=1, prefix="m."),
               "mamba of fives": lambda: Mamba2(D, 10, dv, d, 2, 3, norm_parts=1, prefix="m."),
               "gated of threes": lambda: GatedDelta(D, 6, 2, d, dv, taps, prefix="m.")}[kind]()


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("d,dv,lens", [(64, 64, [48]), (128, 48, [9, 1, 49]), (30, 17, [50, 7]), (200, 20, [16, 63]),
                                       (96, 130, [51]), (7, 3, [1, 2, 3, 4, 5, 11] * 7), (256, 16, [40, 0, 18])])
def test_portions_in_turns_match_single_tokens(kind, d, dv, lens):
    _compare(kind, d, dv, lens, 3)


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("d,dv,lens,turns", [(64, 64, [1, 49, 1, 7, 48], 48), (30, 17, [5, 0, 9, 4, 8, 1] * 6, 5),
                                             (128, 48, [1] * 40 + [50], 50), (96, 20, [3, 2, 1], 48)])
def test_some_requests_in_turns(kind, d, dv, lens, turns):
    """Both ways in one step: requests of at least ``turns`` tokens in turns, the others token by token."""
    _compare(kind, d, dv, lens, 3, turns)


@pytest.mark.parametrize("kind", ["gated", "channel"])
@pytest.mark.parametrize("taps", [2, 4, 6])
@pytest.mark.parametrize("d,dv,lens", [(64, 48, [9, 1, 49, 2]), (30, 17, [50, 7]), (136, 8, [48, 5])])
def test_convolutions_of_turns(kind, taps, d, dv, lens):
    """Rows and coefficients of turns are made with the convolution: filters up to four taps from registers, longer ones beside."""
    _compare(kind, d, dv, lens, taps)


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("d,dv,lens", [(64, 64, [16, 17, 15, 1, 33]), (36, 20, [31, 32, 48, 2]), (128, 4, [50]), (4, 16, [16, 5] * 20),
                                       (100, 132, [35, 0, 64]), (60, 60, [97])])
def test_chunks_at_their_edges(kind, d, dv, lens):
    """Heads that chunks of sixteen tokens take (csrc/state_chunks.cuh): whole and broken chunks, requests between others' places,
    channels and columns that fill no tile."""
    _compare(kind, d, dv, lens, 4)


class _in_turns:
    """The step's requests of at least ``turns`` tokens are walked in turns, whatever the rule says."""

    def __init__(self, turns):
        self.turns = turns

    def __enter__(self):
        from llm_rs_b200 import ops
        self.rule, ops.walk_from = ops.walk_from, lambda *a, **k: self.turns

    def __exit__(self, *a):
        from llm_rs_b200 import ops
        ops.walk_from = self.rule


def _compare(kind, d, dv, lens, taps, turns=1):
    from llm_rs_b200.parts import Runtime
    g = torch.Generator().manual_seed(d + dv)
    D, part = _part(kind, d, dv, taps)
    w = {s.name: (torch.randn(s.shape, generator=g) * (0.5 if len(s.shape) == 1 else s.shape[-1] ** -0.5)).to(DEV)
         for s in part.weight_specs()}
    part.bind(w, Runtime(torch.device(DEV), torch.float32, 4096))
    x = [torch.randn(n, D, generator=g).to(DEV) for n in lens]
    start = {name: 0.3 * torch.randn(len(lens), *shape, generator=g).to(DEV)
             for name, shape in part.state_need().tensors.items()}
    whole = {k: t.clone() for k, t in start.items()}
    with _in_turns(turns):
        got = part.forward(torch.cat(x), _ctx(lens, [0] * len(lens)), SimpleNamespace(state=whole))
    single = {k: t.clone() for k, t in start.items()}
    rows = [[] for _ in lens]
    for i in range(max(lens)):
        n_new = [int(i < n) for n in lens]
        y = part.forward(torch.cat([a[i:i + 1] for a in x if i < a.size(0)]), _ctx(n_new, [min(i, n) for n in lens]),
                         SimpleNamespace(state=single))
        for r, row in zip([r for r, n in enumerate(lens) if i < n], y):
            rows[r].append(row)
    want = torch.stack([row for r in rows for row in r])
    for name, a, b in [("output", got, want)] + [(k, whole[k], single[k]) for k in whole]:
        assert torch.isfinite(a).all(), name
        assert float((a - b).abs().max()) <= 3.2e-5 * max(1.0, float(b.abs().max())), name


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("at", [0, 1, 2, 3, 4, 7, 8, 15, 16, 31, 32, 47, 48, 53, 61])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("d,dv", [(64, 48), (30, 17)])
def test_tokens_before_one_that_is_not_finite_keep_their_numbers(kind, d, dv, at, bad):
    """Wherever the token lies in its chunk (heads of 64) or in its turn (of 30), earlier outputs keep every bit, and its own is no
    number."""
    from llm_rs_b200.parts import Runtime
    g = torch.Generator().manual_seed(3)
    D, part = _part(kind, d, dv)
    w = {s.name: (torch.randn(s.shape, generator=g) * (0.5 if len(s.shape) == 1 else s.shape[-1] ** -0.5)).to(DEV)
         for s in part.weight_specs()}
    part.bind(w, Runtime(torch.device(DEV), torch.float32, 4096))
    x = torch.randn(62, D, generator=g).to(DEV)
    outs = []
    for rows in (x, x.index_fill(0, torch.tensor([at], device=DEV), bad)):
        state = {name: torch.zeros(1, *shape, device=DEV) for name, shape in part.state_need().tensors.items()}
        with _in_turns(1):
            outs.append(part.forward(rows, _ctx([62], [0]), SimpleNamespace(state=state)))
    want, got = outs
    assert torch.isfinite(want).all()
    assert torch.equal(got[:at], want[:at])
    assert not torch.isfinite(got[at]).any()


def _both_ways(kind, d, dv, lens, change_weights, change_x, change_state):
    """(outputs, states) walked and token by token, the step's requests all one way."""
    from llm_rs_b200.parts import Runtime
    g = torch.Generator().manual_seed(7 * d + dv)
    D, part = _part(kind, d, dv)
    w = {s.name: torch.randn(s.shape, generator=g) * (0.5 if len(s.shape) == 1 else s.shape[-1] ** -0.5) for s in part.weight_specs()}
    change_weights(w)
    part.bind({k: t.to(DEV) for k, t in w.items()}, Runtime(torch.device(DEV), torch.float32, 4096))
    x = torch.randn(sum(lens), D, generator=g)
    change_x(x)
    start = {name: 0.3 * torch.randn(len(lens), *shape, generator=g) for name, shape in part.state_need().tensors.items()}
    change_state(start)
    got = []
    for turns in (1, 0):
        state = {k: t.to(DEV) for k, t in start.items()}
        with _in_turns(turns):
            got.append((part.forward(x.to(DEV), _ctx(lens, [0] * len(lens)), SimpleNamespace(state=state)).cpu(),
                        {k: t.cpu() for k, t in state.items()}))
    return got


LINEAR = ("memory", "retention", "mamba")


def _same_kinds_of_numbers(kind, walked, single):
    """Every state finite where it is finite token by token, there the same to float32's rounding (by columns: one of numbers near the
    largest has neighbours of ordinary ones); under a linear rule infinities where they are, with their signs."""
    for name in single:
        a, b = walked[name].double(), single[name].double()
        assert torch.equal(a.isfinite(), b.isfinite()), name
        if kind in LINEAR:
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a[a.isinf()], b[b.isinf()]), name
        a, b = a.nan_to_num(0.0, 0.0, 0.0), b.nan_to_num(0.0, 0.0, 0.0)
        size = b.abs().amax(-2, keepdim=True) if b.dim() > 3 else b.abs().amax()
        assert bool(((a - b).abs() <= 3.2e-5 * size.clamp(min=1.0)).all()), name


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("d,dv", [(64, 48), (36, 20), (30, 17)])
@pytest.mark.parametrize("value", [3.4e38, -1.8e38, float("inf"), float("nan")])
def test_states_at_the_edge_of_the_range(kind, d, dv, value):
    """A state that is huge, infinite or no number in one column: its column alone holds it, in whole and broken chunks."""
    if kind == "general":
        dv = d
    def change(state):
        name = [k for k in state if k.endswith(".state")][0]
        for slot in range(state[name].size(0)):
            state[name][slot, 1, 5 + slot, 3 + slot] = value
    (out, walked), (want, single) = _both_ways(kind, d, dv, [37, 5, 16], lambda w: None, lambda x: None, change)
    _same_kinds_of_numbers(kind, walked, single)
    if abs(value) < 1e39 and d % 4 == 0:      # (in turns a product of three numbers near the range's end is taken in another order)
        assert torch.equal(out.isfinite(), want.isfinite())
        assert float((out - want).nan_to_num(0.0, 0.0, 0.0).abs().max()) <= 3.2e-5 * max(1.0, float(want.nan_to_num(0.0, 0.0, 0.0).abs().max()))


@pytest.mark.parametrize("kind", ["memory", "retention", "gated", "channel", "general"])
@pytest.mark.parametrize("d,dv", [(64, 48), (36, 20), (30, 17)])
@pytest.mark.parametrize("at", [0, 3, 15, 16, 36, 38])
@pytest.mark.parametrize("value", [1.8e38, float("inf")])
def test_values_at_the_edge_of_the_range(kind, d, dv, at, value):
    """A token whose value is huge or infinite in one column, at the first and last token of chunks and of requests."""
    if kind == "general":
        dv = d
    def weights(w):
        w["m.k"] *= 0.2
        w["m.v"][5] = 0.0
        w["m.v"][5, 0] = 1e38
        if "m.v.conv" in w:
            w["m.v.conv"][5] = 1.0
    def tokens(x):
        x[:, 0] = 0.0
        x[at, 0] = value / 1e38
    (_, walked), (_, single) = _both_ways(kind, d, dv, [37, 5, 16], weights, tokens, lambda state: None)
    _same_kinds_of_numbers(kind, walked, single)


@pytest.mark.parametrize("kind", ["memory", "retention", "mamba", "gated", "channel", "general"])
@pytest.mark.parametrize("lens", [[1] * 40 + [50] + [1] * 30 + [0, 49, 48] + [1] * 9 + [97], [0, 0, 48, 47, 64, 1], [1] * 33 + [48]])
def test_walked_requests_among_many_short_ones(kind, lens):
    """The places of chunks are counted over the walked requests alone, 32 requests at a time."""
    _compare(kind, 64, 48, lens, 3, 48)


@pytest.mark.parametrize("kind", ["mamba of one group", "mamba of fives", "gated of threes"])
@pytest.mark.parametrize("d,dv,lens", [(64, 64, [40, 16, 1]), (128, 20, [33]), (64, 16, [17] * 90), (36, 16, [17] * 170)])
def test_heads_that_share_a_key_head(kind, d, dv, lens):
    """Two heads a block of rows, four and all: the last block of a key head has what is left."""
    _compare(kind, d, dv, lens, 3)
