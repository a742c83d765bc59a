"""Which tokens of a step latent attention takes which way (parts/latent_attention.py): plans, made on the host."""
import numpy as np
import pytest


def _ranges(lens, longs):
    from llm_rs_b200.parts.latent_attention import other_ranges
    n_new = np.asarray(lens, np.int64)
    q_start = np.concatenate([[0], np.cumsum(n_new)[:-1]])
    return other_ranges(q_start, n_new, np.asarray(longs, bool), int(n_new.sum()))


@pytest.mark.parametrize("lens,longs,want", [
    ([5], [0], ((0, 5),)), ([300], [1], ()), ([1] * 8 + [1700], [0] * 8 + [1], ((0, 8),)), ([1700] + [1] * 8, [1] + [0] * 8, ((1700, 1708),)),
    ([3, 1000, 4, 2000, 5], [0, 1, 0, 1, 0], ((0, 3), (1003, 1007), (3007, 3012))),
    ([3, 100, 4, 2000, 5], [0, 1, 0, 1, 0], ((0, 107), (2107, 2112))),      # a short gap is taken along
    ([400, 500, 0, 7], [1, 1, 0, 0], ((900, 907),)), ([400, 0, 500], [1, 0, 1], ())])
def test_tokens_of_no_long_portion(lens, longs, want):
    """The folded form's products run over these tokens only: not over a long portion's, which has its own."""
    assert _ranges(lens, longs) == want


def test_a_portion_that_does_not_fit_leaves_the_room_to_others(monkeypatch):
    from llm_rs_b200 import ops
    from llm_rs_b200.parts.latent_attention import expanded_rows
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 1024 * 100)
    n_new, cached = np.array([500, 2000, 128, 300], np.int64), np.zeros(4, np.int64)
    first, counts, is_long = expanded_rows(n_new, cached, 0, 100)
    assert is_long.tolist() == [True, False, True, True]
    assert counts.tolist() == [512, 0, 128, 384] and first.tolist() == [0, 0, 0, 0]
    monkeypatch.setattr(ops, "LATENT_EXPAND_BYTES", 1024 * 100 - 1)
    assert expanded_rows(n_new, cached, 0, 100)[2].tolist() == [True, False, True, False]


@pytest.mark.parametrize("n_new,want", [([64], [1]), ([64, 64], [1, 1]), ([1] * 63 + [64], [0] * 64), ([1, 319], [0, 0]), ([1, 320], [0, 1]),
                                        ([200, 1, 120], [1, 0, 1]), ([200, 1, 119], [0, 0, 0]), ([64, 0], [1, 0]), ([20, 64], [0, 0])])
def test_portions_beside_other_tokens_need_more_of_them(n_new, want):
    from llm_rs_b200.parts.latent_attention import expanded_rows
    n_new = np.asarray(n_new, np.int64)
    assert expanded_rows(n_new, np.zeros_like(n_new), 0, 100)[2].tolist() == [bool(w) for w in want]


@pytest.mark.parametrize("n_new,cached,window,want", [(63, 0, 0, False), (64, 0, 0, True), (32, 32, 0, True), (32, 31, 0, False),
                                                      (40, 1000, 8, True), (31, 500, 0, False)])
def test_portions_over_few_keys_stay_folded(n_new, cached, window, want):
    from llm_rs_b200.parts.latent_attention import expanded_rows
    assert expanded_rows(np.array([n_new]), np.array([cached]), window, 100)[2].tolist() == [want]
