"""The grouped and batched products on tcgen05 (csrc/gemm_grouped_tc.cu) at the edges of their tiles against float64 and the
mma.sync kernel: rows picked by an index or as they lie, groups of no, one, 128 and 129 rows, widths and depths that fill no
tile, the gated unit, both output types; a wait that runs out. Products of bfloat16 numbers are exact in float32, so an output
errs by at most K + 1 half ulps of the sum of the products' magnitudes, and half an ulp of its own type."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bound(x, w, out_dtype, K):
    mag = x.double().abs() @ w.double().abs().t()
    return mag * (K + 1) * 2.0 ** -24 + (mag * 2.0 ** -8 if out_dtype == torch.bfloat16 else 0.0) + 1e-30


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gather", [True, False])
@pytest.mark.parametrize("N,K,counts", [(256, 64, [129, 0, 1, 128, 300]), (200, 72, [500, 20]), (1000, 136, [7, 257, 130]),
                                        (64, 512, [384]), (33, 200, [128, 128, 5])])
def test_grouped(N, K, counts, gather, out_dtype):
    from llm_rs_b200 import ops
    torch.manual_seed(N + K)
    G, rows = len(counts), sum(counts)
    w = torch.randn(G, N, K, device=DEV).bfloat16()
    x = torch.randn(150 if gather else rows, K, device=DEV).bfloat16()
    src = torch.randint(0, x.size(0), (rows,), device=DEV, dtype=torch.int32) if gather else None
    starts = [sum(counts[:g]) for g in range(G)]
    tiles = [(g, s + a, min(128, n - a)) for g, (s, n) in enumerate(zip(starts, counts)) for a in range(0, n, 128)]
    n_tiles = torch.tensor([len(tiles)], dtype=torch.int32, device=DEV)
    tiles = torch.tensor(tiles + [(0, 0, 0)] * 3, dtype=torch.int32, device=DEV)
    out = torch.full((rows, N), 7.0, device=DEV, dtype=out_dtype)
    ops.gemm_grouped(x, w, out, tiles, n_tiles, src, tile_rows=128)
    ops.check_tc_error(DEV)
    rows_x = x[src.long()] if gather else x
    for g, (s, n) in enumerate(zip(starts, counts)):
        want = rows_x[s:s + n].double() @ w[g].double().t()
        assert bool(((out[s:s + n].double() - want).abs() <= _bound(rows_x[s:s + n], w[g], out_dtype, K)).all()), g
    # The gated unit of two products against the other kernel's: float32 sums in another order, rounded once.
    w2 = torch.randn(G, N, K, device=DEV).bfloat16()
    got, other = torch.empty(rows, N, device=DEV), torch.empty(rows, N, device=DEV)
    ops.gemm_grouped(x, w, got, tiles, n_tiles, src, w2=w2, limit=7.0, alpha=1.702, shift=1.0, tile_rows=128)
    ops.grouped_use_tcgen05(False)
    try:
        ops.gemm_grouped(x, w, other, tiles, n_tiles, src, w2=w2, limit=7.0, alpha=1.702, shift=1.0, tile_rows=128)
    finally:
        ops.grouped_use_tcgen05(True)
    ops.check_tc_error(DEV)
    # gate and up each err by some 1e-6 of sqrt(K); the unit multiplies them (gate clamped at 7, up at 7 and shifted).
    assert float((got - other).abs().max()) <= 1e-4 * max(1.0, float(other.abs().max()))


@pytest.mark.parametrize("M,B,N,K,pad", [(128, 3, 128, 64, 0), (129, 4, 512, 128, 8), (300, 2, 40, 192, 16), (2000, 16, 128, 512, 0),
                                         (130, 3, 96, 72, 8)])
def test_batched(M, B, N, K, pad):
    """(K = 72 is no whole number of steps: the mma.sync kernel keeps it.)"""
    from llm_rs_b200 import ops
    torch.manual_seed(M + N)
    wide = torch.randn(M, B * (K + pad) + pad, device=DEV).bfloat16()
    x = wide[:, : B * (K + pad)].unflatten(1, (B, K + pad))[:, :, :K]
    wide[:, B * (K + pad):] = float("nan")      # what lies beside the batches must not be read into a sum
    w = torch.randn(B, N, K, device=DEV).bfloat16()
    out = torch.full((M, B, N + pad), 3.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm_batched(x, w, out[:, :, :N])
    ops.check_tc_error(DEV)
    for b in range(B):
        want = x[:, b].double() @ w[b].double().t()
        assert bool(((out[:, b, :N].double() - want).abs() <= _bound(x[:, b], w[b], torch.bfloat16, K)).all()), b
    assert bool((out[:, :, N:] == 3.0).all())


@pytest.mark.parametrize("M,B,N,K,form", [(128, 3, 128, 64, "batch"), (300, 2, 40, 192, "batch"), (257, 4, 96, 128, "batch"),
                                          (130, 3, 64, 64, "same rows"), (200, 5, 64, 128, "overlapping"), (129, 1, 64, 64, "batch")])
def test_batched_in_other_orders(M, B, N, K, form):
    """Batches one behind the other, the same rows for every batch, rows that overlap: any strides are taken."""
    from llm_rs_b200 import ops
    torch.manual_seed(M + N)
    if form == "batch":
        x = torch.randn(B, M, K, device=DEV).bfloat16().transpose(0, 1)
    elif form == "same rows":
        x = torch.randn(M, 1, K, device=DEV).bfloat16().expand(M, B, K)
    else:
        x = torch.randn(M * 64 + B * 64 + K, device=DEV).bfloat16().as_strided((M, B, K), (64, 64, 1))
    w = torch.randn(B, N, K, device=DEV).bfloat16()
    out = torch.empty((B, M, N), device=DEV, dtype=torch.bfloat16).transpose(0, 1)
    ops.gemm_batched(x, w, out)
    ops.check_tc_error(DEV)
    for b in range(B):
        want = x[:, b].double() @ w[b].double().t()
        assert bool(((out[:, b].double() - want).abs() <= _bound(x[:, b], w[b], torch.bfloat16, K)).all()), b


@pytest.mark.parametrize("tail", [[-1, 1 << 30], []])
def test_rows_that_no_tile_names_need_no_source(tail):
    """Rows are gathered ahead of the tcgen05 kernel: those past the tiles may name no row of X, or have no entry."""
    from llm_rs_b200 import ops
    torch.manual_seed(4)
    x, w = torch.randn(20, 64, device=DEV).bfloat16(), torch.randn(1, 96, 64, device=DEV).bfloat16()
    src = torch.tensor([19, 0, 7] + tail, dtype=torch.int32, device=DEV)
    tiles, n_tiles = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([[0, 0, 3]], [1]))
    out = torch.full((5, 96), 7.0, device=DEV)
    ops.gemm_grouped(x, w, out, tiles, n_tiles, src, tile_rows=128)
    ops.check_tc_error(DEV)
    rows = x[[19, 0, 7]]
    assert bool(((out[:3].double() - rows.double() @ w[0].double().t()).abs() <= _bound(rows, w[0], torch.float32, 64)).all())
    assert bool((out[3:] == 7.0).all())


def test_one_row_of_any_stride():
    from llm_rs_b200 import ops
    x = torch.randn(1, 64, device=DEV).bfloat16()
    w = torch.randn(2, 96, 64, device=DEV).bfloat16()
    tiles, n_tiles = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([[1, 0, 1]], [1]))
    out = torch.empty(1, 96, device=DEV)
    for stride in (8, 64, 1 << 40):
        ops.gemm_grouped(x.as_strided((1, 64), (stride, 1)), w, out, tiles, n_tiles, None, tile_rows=128)
        ops.check_tc_error(DEV)
        want = x.double() @ w[1].double().t()
        assert bool(((out.double() - want).abs() <= _bound(x, w[1], torch.float32, 64)).all())


def test_a_wait_that_runs_out_is_reported():
    from llm_rs_b200 import ops
    x, w = torch.randn(256, 256, device=DEV).bfloat16(), torch.randn(1, 256, 256, device=DEV).bfloat16()
    out = torch.empty(256, 1, 256, device=DEV, dtype=torch.bfloat16)
    ops.set_tc_wait_limit(2000)
    ops.test_skip_copy(gemm_k_block=2)
    try:
        ops.gemm_batched(x.unflatten(1, (1, 256)), w, out)
        with pytest.raises(ops.KernelError, match="gave up waiting"):
            ops.check_tc_error(DEV)
    finally:
        ops.test_skip_copy()
        ops.set_tc_wait_limit()
    ops.gemm_batched(x.unflatten(1, (1, 256)), w, out)
    ops.check_tc_error(DEV)
    assert torch.allclose(out[:, 0].float(), x.float() @ w[0].float().t(), atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,K,counts", [(64, 64, [1]), (200, 72, [3, 0, 29]), (33, 200, [16, 15]), (96, 8, [32]), (130, 136, [33, 1]),
                                        (256, 512, [1] * 20), (65, 328, [64, 5])])
def test_grouped_few_rows(N, K, counts, out_dtype):
    """Tiles of 64 rows on mma.sync in steps of 64 of k, of 32 rows where the list has no more; beside the CUDA-core kernel."""
    from llm_rs_b200 import ops
    torch.manual_seed(N + K)
    G, rows = len(counts), sum(counts)
    w, w2 = (torch.randn(G, N, K, device=DEV).bfloat16() for _ in range(2))
    x = torch.randn(9, K, device=DEV).bfloat16()
    src = torch.randint(0, 9, (rows,), device=DEV, dtype=torch.int32)
    starts = [sum(counts[:g]) for g in range(G)]
    tiles = [(g, s + a, min(64, n - a)) for g, (s, n) in enumerate(zip(starts, counts)) for a in range(0, n, 64)]
    n_tiles = torch.tensor([len(tiles)], dtype=torch.int32, device=DEV)
    tiles = torch.tensor(tiles + [(0, 0, 0)] * 2, dtype=torch.int32, device=DEV)
    out = torch.full((rows, N), 7.0, device=DEV, dtype=out_dtype)
    ops.gemm_grouped(x, w, out, tiles, n_tiles, src, tile_rows=64)
    for g, (s, n) in enumerate(zip(starts, counts)):
        rows_x = x[src[s:s + n].long()]
        want = rows_x.double() @ w[g].double().t()
        assert bool(((out[s:s + n].double() - want).abs() <= _bound(rows_x, w[g], out_dtype, K)).all()), g
    got, other = torch.empty(rows, N, device=DEV), torch.empty(rows, N, device=DEV)
    for on, to in ((True, got), (False, other)):
        ops.grouped_use_tensor_cores(on)
        try:
            ops.gemm_grouped(x, w, to, tiles, n_tiles, src, w2=w2, limit=7.0, alpha=1.702, shift=1.0, tile_rows=64)
        finally:
            ops.grouped_use_tensor_cores(True)
    assert float((got - other).abs().max()) <= 1e-4 * max(1.0, float(other.abs().max()))


@pytest.mark.parametrize("top,width,n", [(1, 4, 3), (4, 2048, 5), (5, 516, 2), (9, 1028, 1), (2, 30, 4)])
@pytest.mark.parametrize("form", ["plain", "plain bf16", "shared", "shared gated bf16", "residual"])
def test_combine(top, width, n, form):
    """Sums of top + 2 products in float32 (an ulp each of the magnitudes) and one rounding of a bfloat16 output; a width of no
    whole pieces takes the other kernel."""
    from llm_rs_b200 import ops
    torch.manual_seed(top + width)
    rows = torch.randn(n * top, width, device=DEV)
    row_of = torch.randperm(n * top, device=DEV).to(torch.int32)
    weight = torch.rand(n * top, device=DEV)
    parts = [(weight[t * top + k].double() * rows[row_of[t * top + k].long()].double()) for t in range(n) for k in range(top)]
    parts = torch.stack(parts).view(n, top, width)
    want, mag = parts.sum(1), parts.abs().sum(1)
    rounding = 0.0
    if form.startswith("plain"):
        dtype = torch.bfloat16 if "bf16" in form else torch.float32
        got = ops.moe_combine(rows, row_of, weight, top, dtype) if dtype == torch.bfloat16 else ops.moe_combine(rows, row_of, weight, top)
        rounding = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    else:
        shared = torch.randn(n, width, device=DEV).to(torch.bfloat16 if "bf16" in form else torch.float32)
        gate = torch.randn(n, 3, device=DEV)[:, 1] if "gated" in form else None
        own = shared.double() * (torch.sigmoid(gate.double())[:, None] if gate is not None else 1.0)
        want, mag = want + own, mag + own.abs()
        if form == "residual":
            got = torch.randn(n, width, device=DEV)
            want, mag = want + got.double(), mag + got.double().abs()
            ops.moe_combine_shared(rows, row_of, weight, top, shared, gate, residual=got)
        else:
            got = ops.moe_combine_shared(rows, row_of, weight, top, shared, gate)
    assert bool(((got.double() - want).abs() <= mag * (top + 4) * 2.0 ** -24 + rounding * want.abs() + 1e-30).all())
