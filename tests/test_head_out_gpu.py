"""The output stage that the recurrent mixers share (csrc/head_out.cuh) and the rows' preparation by pieces, against float64."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dv,heads,n,pad", [(128, 3, 5, 0), (64, 5, 33, 4), (16, 7, 9, 8), (4, 1, 1, 0), (24, 2, 3, 0), (128, 2, 3, 1)])
@pytest.mark.parametrize("normaliser,silu", [(False, True), (True, False)])
def test_linear_recurrence_by_pieces(dtype, dv, heads, n, pad, normaliser, silu):
    """One token a request, decay 0 and state 0, so o = (q . k) b v; the rows may lie on no boundary (pad 1). Inputs are exact;
    float32 sums of at most 16 products and the final rounding to the activation type (2^-8 of it, bfloat16) bound the error."""
    from llm_rs_b200 import ops
    torch.manual_seed(dv + heads + n)
    dk = 8
    width = heads * (2 * dk + 2 * dv)
    rows = torch.randn(n, width + pad, device=DEV).to(dtype)[:, pad:]
    q, k, v, gate = rows.split([heads * dk, heads * dk, heads * dv, heads * dv], dim=1)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    work = {}
    ctx = SimpleNamespace(n_tokens=n, n_requests=n, q_start=i32(list(range(n))), n_new=i32([1] * n), slot_ids=i32(list(range(n))),
                          positions=i32([0] * n), token_req=i32(list(range(n))),
                          scratch=lambda name, f: work.setdefault(name, torch.zeros(f, device=DEV)))
    state = torch.zeros(n, heads, dk, dv, device=DEV)
    norm = torch.zeros(n, heads, dk, device=DEV) if normaliser else None
    gain, floor = torch.rand(n, heads, device=DEV) + 0.5, torch.rand(n, heads, device=DEV)
    w = torch.rand(heads * dv, device=DEV) + 0.5
    got = ops.linear_recurrence(q, k, v, gate, w, state, ctx, heads, dk, dv, 1e-6, decay=torch.zeros(n, heads, device=DEV), gain=gain,
                                normaliser=norm, floor=floor if normaliser else None, den_eps=1e-6, gate_silu=silu)
    d = lambda t, c: t.double().unflatten(1, (heads, c))
    s = (d(q, dk) * d(k, dk)).sum(-1, keepdim=True) * gain.double()[..., None]
    o = s * d(v, dv)
    if normaliser:
        o = o / (torch.maximum(s.abs(), floor.double()[..., None]) + 1e-6)
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * w.double().view(heads, dv)
    g = d(gate, dv)
    want = (o * (g if silu else 1.0) * torch.sigmoid(g)).flatten(1)
    # q . k may cancel: its float32 error relative to it is 2^-21 of sum |q k| over it.
    loss = ((d(q, dk) * d(k, dk)).abs().sum(-1, keepdim=True) / (d(q, dk) * d(k, dk)).sum(-1, keepdim=True).abs())
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) + 2.0 ** -18 + 2.0 ** -21 * loss.expand(-1, -1, dv).flatten(1)
    assert bool(((got.double() - want).abs() <= bound * want.abs() + 1e-6).all())
