"""The gates' scan (csrc/linear_recurrence.cu) of portions against float64."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("portions,heads", [([128], 3), ([129, 1, 7], 4), ([70, 60], 4), ([300, 2049], 5), ([4100], 2), ([2048, 8], 1),
                                            ([1] * 40 + [130, 127, 0, 128], 19), ([2] * 130, 17)])
def test_scan_in_runs(portions, heads):
    """|m| stays below 64 here, so that a rounding of it is at most 2^-19, and f and i (at most 15, from tanhf) are off by 2^-20
    at most. A maximum carries the roundings since the last token that set it: sixteen of them are allowed for, 2^-15."""
    from llm_rs_b200 import ops
    torch.manual_seed(sum(portions) + heads)
    cap, n = 15.0, sum(portions)
    gates = torch.randn(n, 2 * heads + 3, device=DEV)[:, : 2 * heads] * 6
    gates[:, heads:] += 3
    slots = list(range(len(portions)))[::-1]
    m0 = torch.randn(len(portions), heads, device=DEV) * 3
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    starts = [sum(portions[:r]) for r in range(len(portions))]
    m = m0.clone()
    got = ops.gate_scan(gates, cap, m, SimpleNamespace(q_start=i32(starts), n_new=i32(portions), slot_ids=i32(slots),
                                                       n_requests=len(portions)), heads)
    g = gates.cpu().double()
    i, f = cap * torch.tanh(g[:, :heads] / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(g[:, heads:] / cap))
    bound = 2.0 ** -15
    for r, (a, k) in enumerate(zip(starts, portions)):
        state = m0[slots[r]].cpu().double()
        for t in range(a, a + k):
            new = torch.maximum(f[t] + state, i[t])
            assert float(new.abs().max()) < 64
            for have, want in zip(got, (torch.exp(f[t] + state - new), torch.exp(i[t] - new), torch.exp(-new))):
                assert bool(((have[t].cpu().double() - want).abs() <= bound * want + 1e-30).all())
            state = new
        assert bool(((m[slots[r]].cpu().double() - state).abs() <= bound).all())


def test_a_requests_numbers_do_not_depend_on_the_step():
    """A request alone, beside a portion, and with the step's lengths known to the host: the same bits."""
    from llm_rs_b200 import ops
    torch.manual_seed(2)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lens, heads = [7, 300, 1, 100, 128], 11
    gates, m0 = torch.randn(sum(lens), 2 * heads, device=DEV) * 4, torch.randn(len(lens), heads, device=DEV)

    def run(which, host):
        starts = [sum(lens[:r]) for r in range(len(lens))]
        rows = torch.cat([gates[starts[r]: starts[r] + lens[r]] for r in which])
        k, m = [lens[r] for r in which], m0[which].clone()
        ctx = SimpleNamespace(q_start=i32([sum(k[:j]) for j in range(len(k))]), n_new=i32(k), slot_ids=i32(list(range(len(k)))),
                              n_requests=len(k), host_n_new=k if host else None)
        return [torch.split(t, k) for t in ops.gate_scan(rows.contiguous(), 9.0, m, ctx, heads)] + [list(m)]
    whole = run(list(range(len(lens))), True)
    assert all(torch.equal(a, b) for x, y in zip(whole, run(list(range(len(lens))), False)) for a, b in zip(x, y))
    for r in range(len(lens)):
        assert all(torch.equal(x[r], y[0]) for x, y in zip(whole, run([r], True))), lens[r]
