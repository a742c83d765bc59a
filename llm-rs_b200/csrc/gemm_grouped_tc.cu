// The grouped and batched products of gemm_grouped.cu for many rows, on tcgen05: out[row, n] = sum_k X[src(row), k] *
// W_g[n, k], or the gated unit of two such products. bfloat16 operands, float32 sums in order of k: a row's result does not
// depend on which rows share its tile.
//
// One block per SM walks tiles of 128 rows x 256 columns (the gated unit: 128 columns of each of its two weights; 128 columns
// where N is no more). Warp 0 copies by TMA: the rows of X as they lie (rows m0 .. m0 + 127 of a batch; rows beyond a group's
// end belong to the next one and are not stored), the weights as one tensor of groups * N rows. Rows that `src` picks are
// gathered beforehand (gather_rows): picked by the copy itself, four rows an instruction (tile::gather4), a stage of 128 rows
// took 32 copies and the gated product of 8,192 rows some 200 us instead of what it takes now. Warp 1 issues the MMAs, warps
// 2-5 run the epilogue on an accumulator that is double-buffered in tensor memory, so that a tile's stores run under the next
// tile's MMAs. Tiles that share weights are neighbours in the walk: the blocks that run together read one group's weights
// from the L2.
//
// 8,192 rows in 32 groups, K = 2,048, gated into 1,024 columns: 107 us (303 with mma.sync tiles of 128 x 64 x 2, bound by the
// shared-memory reads of their fragments); K = 1,024 into 2,048 columns of float32: 58 us (163). The weights' stream is 41 and
// 21 us of that; what bounds it now is the copies of the tiles, 48 KB a step of k and block, from the L2. gemm_grouped.cu keeps
// small groups and rows that TMA cannot address.
//
// Every wait is bounded (see gemm_tcgen05.cu): a block that gives up drains its copies and MMAs, records a code in
// *error_flag, frees its tensor memory and returns.
#include "gemm_grouped.cuh"
#include "tcgen05_util.cuh"

uint32_t llmrs_tc_wait_limit();
int llmrs_tc_skipped_copy();

constexpr int GT_STAGES = 4, GT_THREADS = 192, GT_HALF = 128;      // GT_HALF: weight rows of one copy
constexpr uint32_t GT_A_BYTES = TC_BM * TC_BK * 2, GT_HALF_BYTES = GT_HALF * TC_BK * 2;
constexpr uint32_t GT_STAGE_BYTES = GT_A_BYTES + 2 * GT_HALF_BYTES;

struct GtParams {
  void* out;
  long long out_stride, out_batch;
  int out_f32, vec;            // vec: 16-byte stores may be used
  int N, nkb, n_n, glu, halves;
  const int* tiles;            // [tile][3] = group, first row, rows; null: batched
  const int* n_tiles;
  int n_m, M, batches, x_batch;      // batched: tiles of a batch, rows, batches, columns from a batch's rows to the next one's
  GatedUnit unit;
  int* error_flag;
  uint32_t wait_limit;
  int test_skip_kb;
};

// The tile of work item t: group (or batch), first row, rows, first column.
struct GtTile { int group, m0, rows, n0; };
__device__ __forceinline__ GtTile gt_tile(const GtParams& p, int t, int n_row_tiles) {
  const int i = t % n_row_tiles, n = t / n_row_tiles;
  GtTile w;
  if (p.tiles) {
    w.group = p.tiles[3 * i], w.m0 = p.tiles[3 * i + 1], w.rows = p.tiles[3 * i + 2];
  } else {
    w.group = i / p.n_m, w.m0 = i % p.n_m * TC_BM, w.rows = min(TC_BM, p.M - w.m0);
  }
  w.n0 = n * (p.glu ? GT_HALF : p.halves * GT_HALF);
  return w;
}

__global__ void __launch_bounds__(GT_THREADS, 1)
gemm_grouped_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                       const __grid_constant__ CUtensorMap map_w2, const GtParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem + 1023) & ~(uintptr_t)1023);
  // full[4], empty[4], acc_full[2], acc_empty[2], drain
  uint64_t* bars = reinterpret_cast<uint64_t*>(stages + (size_t)GT_STAGES * GT_STAGE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * GT_STAGES + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full0 = tc_smem(bars), empty0 = tc_smem(bars + GT_STAGES), acc_full0 = tc_smem(bars + 2 * GT_STAGES),
                 acc_empty0 = acc_full0 + 16, drain_bar = acc_full0 + 32;
  if (tid == 0) {
    for (int s = 0; s < 2 * GT_STAGES + 2; ++s) mbar_init(full0 + 8 * s, 1);
    mbar_init(acc_empty0, 128);
    mbar_init(acc_empty0 + 8, 128);
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_row_tiles = p.tiles ? *p.n_tiles : p.n_m * p.batches, n_work = n_row_tiles * p.n_n, nkb = p.nkb;
  long long copies = 0;      // warp 0: stages whose copies it has requested

  if (warp == 0) {
    const bool leader = tc_elect_one();
    const uint32_t stage_bytes = GT_A_BYTES + (uint32_t)p.halves * GT_HALF_BYTES;
    long long it = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_work && ok; t += gridDim.x) {
      const GtTile w = gt_tile(p, t, n_row_tiles);
      const int w_row = w.group * p.N + w.n0;
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = (int)(it % GT_STAGES);
        if (it >= GT_STAGES) {
          ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, (uint32_t)((it / GT_STAGES) - 1) & 1, p.wait_limit, abort_flag));
          if (!ok) break;
        }
        if (it != p.test_skip_kb) {
          const uint32_t bar = full0 + 8 * s, a_dst = tc_smem(stages + (size_t)s * GT_STAGE_BYTES);
          if (leader) {
            mbar_expect_tx(bar, stage_bytes);
            tma_load_2d(a_dst, &map_x, bar, kb * TC_BK + (p.tiles ? 0 : w.group * p.x_batch), w.m0);
            tma_load_2d(a_dst + GT_A_BYTES, &map_w, bar, kb * TC_BK, w_row);
            if (p.halves == 2)
              tma_load_2d(a_dst + GT_A_BYTES + GT_HALF_BYTES, p.glu ? &map_w2 : &map_w, bar, kb * TC_BK,
                          p.glu ? w_row : w_row + GT_HALF);
          }
        }
        __syncwarp();
      }
    }
    copies = it;
  } else if (warp == 1) {
    const uint32_t idesc = tc_instr_desc(p.halves * GT_HALF);
    const bool leader = tc_elect_one();
    long long it = 0;
    int lt = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_work && ok; t += gridDim.x, ++lt) {
      const int buf = lt & 1;
      if (lt >= 2) {      // the epilogue has read the tile before last out of this buffer
        ok = __all_sync(0xffffffffu, mbar_wait(acc_empty0 + 8 * buf, (uint32_t)((lt >> 1) - 1) & 1, p.wait_limit, abort_flag));
        if (!ok) break;
        tc_fence_after();
      }
      const uint32_t d_addr = tmem_base + (uint32_t)buf * 256;
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = (int)(it % GT_STAGES);
        ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (uint32_t)(it / GT_STAGES) & 1, p.wait_limit, abort_flag));
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = tc_smem(stages + (size_t)s * GT_STAGE_BYTES);
        const uint64_t a_desc = tc_smem_desc(a_addr), b_desc = tc_smem_desc(a_addr + GT_A_BYTES);
#pragma unroll
        for (int k = 0; k < TC_BK / 16; ++k)
          if (leader) tc_mma(d_addr, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
        if (leader) tc_commit(empty0 + 8 * s);
        __syncwarp();
      }
      if (leader && ok) tc_commit(acc_full0 + 8 * buf);
      __syncwarp();
    }
  } else {
    // Epilogue: a lane of a warp owns a row of the tile; a warp reaches the 32 lanes of tensor memory that its index
    // modulo 4 names.
    const int quarter = warp & 3, r = quarter * 32 + lane;
    int lt = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_work && ok; t += gridDim.x, ++lt) {
      const GtTile w = gt_tile(p, t, n_row_tiles);
      const int buf = lt & 1, width = p.glu ? GT_HALF : p.halves * GT_HALF;
      ok = __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * buf, (uint32_t)(lt >> 1) & 1, p.wait_limit, abort_flag));
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * 256;
      const size_t at = (size_t)(w.m0 + r) * p.out_stride + (p.tiles ? 0 : (size_t)w.group * p.out_batch);
      for (int c = 0; c < width && w.n0 + c < p.N; c += 32) {      // all lanes: the reads are warp-wide
        float v[32];
        tc_ld32(taddr + c, v);
        if (p.glu) {
          float u[32];
          tc_ld32(taddr + GT_HALF + c, u);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = p.unit(v[e], u[e]);
        }
        const int n = w.n0 + c, left = p.N - n;
        if (r >= w.rows) {
          // no row of the tile: nothing to store
        } else if (p.out_f32) {
          float* o = (float*)p.out + at + n;
          if (p.vec && left >= 32) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(o + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (e < left) o[e] = v[e];
          }
        } else {
          __nv_bfloat16* o = (__nv_bfloat16*)p.out + at + n;
          if (p.vec && left >= 32) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint4 pk;
              __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
              for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[e + 2 * i], v[e + 2 * i + 1]);
              *reinterpret_cast<uint4*>(o + e) = pk;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (e < left) o[e] = __float2bfloat16_rn(v[e]);
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty0 + 8 * buf) : "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // The block gave up: the MMAs that were issued must be done, and no copy may still be on its way here.
    if (warp == 1) {
      if (tc_elect_one()) tc_commit(drain_bar);
      __syncwarp();
      mbar_drain(drain_bar, 0, p.wait_limit);
    } else if (tid == 0) {
      for (long long i = copies > GT_STAGES ? copies - GT_STAGES : 0; i < copies; ++i)
        if (i != p.test_skip_kb) mbar_drain(full0 + 8 * (int)(i % GT_STAGES), (uint32_t)(i / GT_STAGES) & 1, p.wait_limit);
      if (p.error_flag) atomicExch(p.error_flag, 1);
    }
    __syncthreads();
  }
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

static int gt_map(CUtensorMap* map, const void* base, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return llmrs_fail("gemm_grouped: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return llmrs_fail("gemm_grouped: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

int launch_grouped_tc(const GroupedGemmArgs& a, int out_dtype, int x_rows, int groups, int batches, int max_tiles,
                      int* error_flag, cudaStream_t stream) {
  GtParams p = {};
  p.out = a.out, p.out_stride = a.out_stride, p.out_batch = a.out_batch, p.out_f32 = out_dtype == LLMRS_F32;
  const long long size = p.out_f32 ? 4 : 2;
  p.vec = ((uintptr_t)a.out & 15) == 0 && a.out_stride * size % 16 == 0 && a.out_batch * size % 16 == 0;
  p.N = a.N, p.nkb = (a.K + TC_BK - 1) / TC_BK, p.glu = a.w2 != nullptr, p.halves = p.glu || a.N > GT_HALF ? 2 : 1;
  const int cols = p.glu ? GT_HALF : p.halves * GT_HALF;
  p.n_n = (a.N + cols - 1) / cols;
  p.tiles = a.tiles, p.n_tiles = a.n_tiles, p.M = a.M, p.batches = batches;
  p.n_m = (a.M + TC_BM - 1) / TC_BM;
  p.unit = a.unit, p.error_flag = error_flag, p.wait_limit = llmrs_tc_wait_limit(), p.test_skip_kb = llmrs_tc_skipped_copy();
  const long long work = (long long)(a.tiles ? max_tiles : p.n_m * batches) * p.n_n;
  LLMRS_REQUIRE(work <= 0x7fffffffLL && (long long)groups * a.N <= 0x7fffffffLL, "gemm_grouped: too many tiles or weights");
  CUtensorMap mx, mw, mw2;
  int rc = 0;
  // All batches are one tensor of wide rows.
  p.x_batch = (int)a.x_batch;
  const cuuint64_t xdims[2] = {(cuuint64_t)(a.tiles ? a.K : (batches - 1) * a.x_batch + a.K), (cuuint64_t)x_rows};
  const cuuint64_t xstrides[1] = {(cuuint64_t)a.x_stride * 2};
  const cuuint32_t xbox[2] = {TC_BK, TC_BM};
  if ((rc = gt_map(&mx, a.x, xdims, xstrides, xbox)) != 0) return rc;
  const cuuint64_t wdims[2] = {(cuuint64_t)a.K, (cuuint64_t)groups * a.N}, wstrides[1] = {(cuuint64_t)a.K * 2};
  const cuuint32_t wbox[2] = {TC_BK, GT_HALF};
  if ((rc = gt_map(&mw, a.w, wdims, wstrides, wbox)) != 0) return rc;
  if ((rc = gt_map(&mw2, a.w2 ? a.w2 : a.w, wdims, wstrides, wbox)) != 0) return rc;
  const size_t smem = 1024 + (size_t)GT_STAGES * GT_STAGE_BYTES + (2 * GT_STAGES + 5) * 8 + 16;
  int dev = 0, n_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  const cudaError_t e = cudaFuncSetAttribute(gemm_grouped_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return llmrs_fail("gemm_grouped: shared memory %zu: %s", smem, cudaGetErrorString(e));
  gemm_grouped_tc_kernel<<<(unsigned)(work < n_sm ? work : (n_sm > 0 ? n_sm : 1)), GT_THREADS, smem, stream>>>(mx, mw, mw2, p);
  return llmrs_launch_status("gemm_grouped (tcgen05)");
}

// out[r] = x[src[r]] for rows of `pieces` 16-byte pieces; a warp per row. A row whose source is none of x's is left as it is: no
// tile may name it, and a list of tiles need not cover all rows.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const uint4* __restrict__ x, long long x_stride, int x_rows, const int* __restrict__ src, uint4* __restrict__ out,
                   int rows, int pieces) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  const int at = src[r];
  if (at < 0 || at >= x_rows) return;
  const uint4* from = x + (size_t)at * x_stride;
  uint4* to = out + (size_t)r * pieces;
#pragma unroll 4
  for (int e = lane; e < pieces; e += 32) to[e] = from[e];
}

// x: x_rows bfloat16 rows of K values, x_stride apart; out [rows, K].
LLMRS_API int llmrs_gather_rows(const void* x, long long x_stride, int x_rows, const int* src, void* out, int rows, int K,
                                cudaStream_t stream) {
  LLMRS_REQUIRE(rows >= 0 && K > 0 && K % 8 == 0 && x_stride % 8 == 0 && (((uintptr_t)x | (uintptr_t)out) & 15) == 0,
                "gather_rows: rows of whole 16-byte pieces");
  if (rows == 0) return 0;
  gather_rows_kernel<<<(rows + 7) / 8, 256, 0, stream>>>((const uint4*)x, x_stride / 8, x_rows, src, (uint4*)out, rows, K / 8);
  return llmrs_launch_status("gather_rows");
}
