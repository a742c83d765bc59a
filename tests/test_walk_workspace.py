"""The workspace of the recurrences with a matrix state: a step that walks no request (decoding, captured in graphs that each hold
their own) has none of the walk's rows, one that walks some has rows for those."""
import pytest

from llm_rs_b200 import ops


def _sizes(tokens, requests, walk_from):
    call = lambda name, *a: int(ops._lib_ll(name)(*a))
    return {"gated": call("llmrs_gated_delta_work_floats", tokens, requests, 8, 16, 128, 128, 0, walk_from),
            "channel": call("llmrs_gated_delta_work_floats", tokens, requests, 16, 16, 128, 128, 1, walk_from),
            "general": call("llmrs_delta_rule_work_floats", tokens, requests, 32, 64, walk_from),
            "linear": call("llmrs_linear_recurrence_work_floats", tokens, requests, 16, 128, 128, walk_from),
            "tables": call("llmrs_linear_recurrence_table_floats", tokens, requests, 16, 128, 128, walk_from)}


@pytest.mark.parametrize("requests", [1, 64, 256])
def test_decode_steps_hold_no_rows_of_a_walk(requests):
    """What the kernels token by token read: q, k, v, read-outs, decays and write strengths of a token."""
    planes = {"gated": 2 * 8 * 128 + 2 * 16 * 128 + 3 * 16, "channel": 2 * 16 * 128 + 2 * 16 * 128 + 16 * 128 + 16, "general": 7 * 32 * 64,
              "linear": 16 * 3 * 128, "tables": 0}
    for kind, size in _sizes(requests, requests, 0).items():
        assert planes[kind] * requests <= size <= planes[kind] * requests + 64, kind


@pytest.mark.parametrize("kind", ["gated", "channel", "general", "linear"])
def test_short_requests_take_no_places(kind):
    """255 single tokens beside a portion of 512, walked alone: what every token needs, and rows (a head's of sixteen tokens: `tile`) of
    the portion and of the places that 255 tokens, and requests of 48 in 767 tokens, can take at most."""
    heads, tile = {"gated": (16, 9920), "channel": (16, 9920), "general": (32, 6976), "linear": (16, 6656)}[kind]
    alone, single = _sizes(512, 1, 48)[kind], _sizes(255, 255, 0)[kind]
    assert _sizes(767, 256, 48)[kind] <= alone + 3 * single + (255 // 16 + 1 + 767 // 48) * heads * tile
    assert _sizes(767, 256, 48)[kind] < _sizes(767, 256, 1)[kind]


def test_portions_walked_by_themselves_hold_no_prepared_rows():
    assert _sizes(8192, 4, 1)["general"] < _sizes(8192, 4, 48)["general"] - 6 * 8192 * 32 * 64 + 64
    for walk_from in (1, 48):      # heads that go in turns of four tokens
        assert int(ops._lib_ll("llmrs_delta_rule_work_floats")(8192, 4, 32, 72, walk_from)) >= 7 * 8192 * 32 * 72
