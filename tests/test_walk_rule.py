"""Which requests of a step the recurrences walk in turns (``ops.walk_from``): a decision of the host alone."""
from types import SimpleNamespace

import pytest

SIZES = dict(gated=dict(blocks=128, least=48, per=32), linear=dict(blocks=144, few=1024), general=dict(blocks=128))


def _walk_from(kind, lens, listed=True):
    from llm_rs_b200 import ops
    ctx = SimpleNamespace(n_requests=len(lens), host_n_new=list(lens) if listed else None)
    return ops.walk_from(ctx, sum(lens), **SIZES[kind])


@pytest.mark.parametrize("kind", list(SIZES))
@pytest.mark.parametrize("lens,want", [
    ([2048], 1), ([48], 1), ([47], 0), ([1], 0), ([1] * 64, 0), ([64] * 8, 1),
    ([2] * 50, 0), ([4] * 24, 0), ([20] * 8, 0), ([47] * 30, 0),      # many short portions: none is worth a walk
    ([1] * 63 + [64], 0), ([1] * 200 + [256], 0),                     # single tokens with a portion that does not pay
    ([1] * 63 + [512], 48), ([1] * 6 + [300, 77], 1)])
def test_lengths_decide(kind, lens, want):
    assert _walk_from(kind, lens) == want
    assert _walk_from(kind, lens[::-1]) == want


@pytest.mark.parametrize("kind", list(SIZES))
def test_without_the_hosts_list_one_portion_is_assumed(kind):
    assert _walk_from(kind, [1311, 1, 1, 402, 1, 77], listed=False) == 1
    assert _walk_from(kind, [1] * 64, listed=False) == 0
    assert _walk_from(kind, [1] * 63 + [64], listed=False) == 0
    assert _walk_from(kind, [2] * 50, listed=False) in (0, 48)      # (at 48 the device finds no request that long)


@pytest.mark.parametrize("channels,d,channel,want", [(512, 64, False, 213), (4096, 128, False, 48), (4096, 128, True, 80),
                                                     (8192, 128, True, 48), (512, 64, True, 375)])
def test_line_of_the_gated_rule(channels, d, channel, want):
    from llm_rs_b200 import ops
    assert ops._gated_walk_least(channels, d, channel) == want
