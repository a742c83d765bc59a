"""How a decode step's keys are cut into runs (``ops.scored_decode_runs``): a decision of the host alone."""
import pytest
import torch


def _runs(span, n_dec=48, heads=16, kv=4, dk=128, dv=None, dtype=torch.bfloat16, q_at=0, q_width=None, cache_at=0):
    from llm_rs_b200 import ops
    q = torch.zeros(n_dec * (q_width or heads * dk) + 8, dtype=dtype)[q_at:].as_strided((n_dec, heads * dk), (q_width or heads * dk, 1))
    cache = torch.zeros(64, dtype=dtype)[cache_at:]
    assert cache.data_ptr() % 16 == 2 * cache_at % 16
    return ops.scored_decode_runs(n_dec, heads, kv, q, cache, dk, dk if dv is None else dv, span)


def test_rows_and_heads_that_the_tensor_cores_do_not_take_are_cut_for_the_other_kernels():
    """None: the caller then cuts the keys for the kernels that will take them."""
    assert _runs(4096) is not None and _runs(4096, dk=64) is not None
    assert _runs(4096, dk=96) is None and _runs(4096, dv=64) is None and _runs(4096, dtype=torch.float32) is None
    assert _runs(4096, cache_at=1) is None and _runs(4096, cache_at=4) is None and _runs(4096, cache_at=8) is not None
    assert _runs(4096, q_at=1) is None and _runs(4096, q_at=2) is not None and _runs(4096, q_width=16 * 128 + 1) is None


@pytest.mark.parametrize("span", [1, 63, 64, 65, 4096, 30001])
@pytest.mark.parametrize("n_dec,heads,kv", [(1, 16, 4), (48, 16, 4), (7, 5, 1), (300, 32, 32)])
def test_runs_cover_the_span(span, n_dec, heads, kv):
    n, keys = _runs(span, n_dec, heads, kv)
    assert keys % 64 == 0 and n * keys >= span > (n - 1) * keys


@pytest.mark.parametrize("n_dec", [1, 48, 64, 256])
@pytest.mark.parametrize("span", [3000, 30000, 131072])
def test_runs_stay_short_however_long_the_longest_request(n_dec, span):
    """The span is the longest request's; the runs of all requests are cut from it."""
    from llm_rs_b200 import ops
    assert _runs(span, n_dec)[1] <= ops.DECODE_RUN_KEYS == 1024
