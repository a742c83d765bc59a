// True 32-bit matrix product for the float32 path: out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]).
//
// FFMA on the CUDA cores, no tensor-core mode of reduced precision. Every output
// element is summed over k in the same order whatever M is, so a token's result does
// not depend on what else is in the batch. The reference's products are library calls
// (llm-core/src/backends/candle.rs:1276-1340: weight [out, in], used transposed,
// optional bias added after).
#include "common.cuh"
#include "mma_util.cuh"

#include <algorithm>
#include <type_traits>

// The order of an output's sum: K falls into segments of GF_SEG values; a segment is one chain of fused multiply-adds in order
// of k, starting at zero, and the segments' sums are added in order, starting at zero. Every kernel below keeps to that order,
// whatever its tile, so an output has the same bits in every batch; and a product of few rows may walk its segments side by
// side, which a single chain over K could not.
constexpr int GF_SEG = 256;

// Four values of a row as floats.
__device__ __forceinline__ float4 gf_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 gf_four(const __nv_bfloat16* p) {
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + 2));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

template <int TM, int TN>
__device__ __forceinline__ void gf_add(float (&acc)[TM][TN], const float4 (&a)[TM], const float4 (&b)[TN]) {
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      acc[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, acc[i][j]))));
}

// The barrier between a round's sums and their readers: of the cluster, or of the block that is alone.
__device__ __forceinline__ void gf_round_arrive(int n_blocks) {
  if (n_blocks > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void gf_round_wait(int n_blocks) {
  if (n_blocks > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  else __syncthreads();
}
// *p in the shared memory of the cluster's block `rank`.
__device__ __forceinline__ float gf_peer(const float* p, int rank, int n_blocks) {
  if (n_blocks == 1) return *p;
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote));      // (volatile: stays behind the barrier)
  return v;
}

// ---------------------------------------------------------------------------------
// Many rows: a block owns a tile of BM rows x BN features and walks K in steps of BK through NS stages of shared memory, filled
// by asynchronous copies NS - 1 steps ahead. Both operands stay in rows along K as they come, a row padded by 16 bytes so that
// neighbouring rows' 16-byte reads fall into different banks; a thread reads four values of K of its TM rows and TN
// features at a time and adds them in order of K. The sums of the segments before lie in registers, or, IN_REGS false, in shared
// memory (each thread its own, touched once in 256 values of K), where a thread's registers are full of operands read ahead.
// Bound by the path from shared memory to registers, 16 reads for 64 multiply-adds, beside the FMA units: 2,048 rows of
// 1,024 into 6,144 features 688 us (37.5 TFLOP/s; 705 as one chain over K, 2,048 x 4,096 x 12,288 5,437 and 5,550).
// ---------------------------------------------------------------------------------
template <typename TX, int BM, int BN, int TM, int TN, int BK, int NS, bool VEC, bool IN_REGS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const TX* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ out, int M, int N, int K, long long x_stride, long long out_stride) {
  constexpr int THREADS = (BM / TM) * (BN / TN), CN = BN / TN, RM = BM / TM;
  constexpr int XS = BK + 16 / (int)sizeof(TX), WS = BK + 4;      // elements a row of a stage takes
  static_assert(GF_SEG % BK == 0, "a step lies in one segment");
  extern __shared__ __align__(16) unsigned char gf_raw[];
  float* tot = reinterpret_cast<float*>(gf_raw);                  // [TM * TN][THREADS]
  float* ws = tot + (IN_REGS ? 0 : TM * TN * THREADS);                 // [NS][BN][WS]
  TX* xs = reinterpret_cast<TX*>(ws + NS * BN * WS);              // [NS][BM][XS]
  const int tid = threadIdx.x, tx = tid % CN, ty = tid / CN;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto load = [&](int stage, int k0) {
    float* wd = ws + stage * BN * WS;
    TX* xd = xs + stage * BM * XS;
    if constexpr (VEC) {      // K, the strides and the bases are multiples of four values: a piece lies inside a row or outside
      for (int e = tid; e < BN * (BK / 4); e += THREADS) {
        const int r = e / (BK / 4), c = e % (BK / 4) * 4;
        const bool in = n0 + r < N && k0 + c < K;
        cp_async_16(wd + r * WS + c, in ? w + (size_t)(n0 + r) * K + k0 + c : w, in ? 16 : 0);
      }
      for (int e = tid; e < BM * (BK / 4); e += THREADS) {
        const int r = e / (BK / 4), c = e % (BK / 4) * 4;
        const bool in = m0 + r < M && k0 + c < K;
        const TX* src = in ? x + (size_t)(m0 + r) * x_stride + k0 + c : x;
        if constexpr (sizeof(TX) == 4) cp_async_16(xd + r * XS + c, src, in ? 16 : 0);
        else cp_async_8(xd + r * XS + c, src, in ? 8 : 0);
      }
    } else {
      // Value by value: a thread keeps to a column and goes down the rows, so that an address is one addition (1,000 rows of
      // 1,023 into 1,024 features 72 us; 141 with an address and plain loads a value; 2,050 into 2,048 276 and 523).
      static_assert(THREADS % BK == 0, "whole rows a pass");
      constexpr int PASS = THREADS / BK;
      const int c = tid % BK, r0 = tid / BK;
      const bool k_in = k0 + c < K;
      const float* wp = w + (size_t)(n0 + r0) * K + k0 + c;
#pragma unroll
      for (int r = 0; r < BN; r += PASS, wp += (size_t)PASS * K) {
        const bool in = k_in && n0 + r0 + r < N;
        if (BN % PASS == 0 || r0 + r < BN) cp_async_4(wd + (r0 + r) * WS + c, in ? wp : w, in ? 4 : 0);
      }
      const TX* xp = x + (size_t)(m0 + r0) * x_stride + k0 + c;
#pragma unroll
      for (int r = 0; r < BM; r += PASS, xp += PASS * x_stride) {
        const bool in = k_in && m0 + r0 + r < M;
        if (BM % PASS == 0 || r0 + r < BM) {
          if constexpr (sizeof(TX) == 4) cp_async_4(xd + (r0 + r) * XS + c, in ? xp : x, in ? 4 : 0);
          else xd[(r0 + r) * XS + c] = in ? *xp : TX(0.f);      // (no asynchronous copy has two bytes)
        }
      }
    }
    cp_async_commit();
  };
  float acc[TM][TN], held[IN_REGS ? TM : 1][IN_REGS ? TN : 1];
  auto before = [&](int i, int j) -> float& {      // the segments before, of this thread's output (i, j)
    if constexpr (IN_REGS) return held[i][j];
    else return tot[(i * TN + j) * THREADS + tid];
  };
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = before(i, j) = 0.f;
  const int steps = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) {
    if (s < steps) load(s, s * BK);
    else cp_async_commit();
  }
  for (int it = 0; it < steps; ++it) {
    cp_async_wait<NS - 2>();
    __syncthreads();      // stage `it` is there for everyone, and everyone is done with the stage that is filled next
    if (it + NS - 1 < steps) load((it + NS - 1) % NS, (it + NS - 1) * BK);
    else cp_async_commit();
    if (it % (GF_SEG / BK) == 0 && it) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          before(i, j) += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
    const float* wr = ws + (it % NS) * BN * WS;
    const TX* xr = xs + (it % NS) * BM * XS;
    if constexpr (IN_REGS && TM * TN > 32) {      // no registers left to read ahead
      float4 av[TM], bv[TN];
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
#pragma unroll
        for (int i = 0; i < TM; ++i) av[i] = gf_four(xr + (ty + i * RM) * XS + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) bv[j] = gf_four(wr + (tx + j * CN) * WS + k);
        gf_add<TM, TN>(acc, av, bv);
      }
    } else {      // the next piece is read while the present one is added
      float4 av[2][TM], bv[2][TN];
      auto fetch = [&](int buf, int k0) {
#pragma unroll
        for (int i = 0; i < TM; ++i) av[buf][i] = gf_four(xr + (ty + i * RM) * XS + k0);
#pragma unroll
        for (int j = 0; j < TN; ++j) bv[buf][j] = gf_four(wr + (tx + j * CN) * WS + k0);
      };
      fetch(0, 0);
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        const int cur = (k / 4) & 1;
        if (k + 4 < BK) fetch(cur ^ 1, k + 4);
        gf_add<TM, TN>(acc, av[cur], bv[cur]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * RM;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * CN;
      if (n < N) out[(size_t)m * out_stride + n] = before(i, j) + acc[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

// ---------------------------------------------------------------------------------
// Few rows, or few tiles: KG groups of RM x CN threads walk KG segments of the block's tile side by side, a thread TM rows x TN
// features of one segment, and the blocks of a cluster take KG segments each. After such a round every sum of a segment lies
// in its block's shared memory, and each block adds its share of the tile over all of them in order. What bounds it: one row
// is the stream of the weights (every one read from shared memory once) and the latency of a launch, a segment's chain being
// 0.6 us; rows that fill TM the path from shared memory to registers, (TM + TN) reads for TM x TN multiply-adds.
// One row: 1,024 into 1,024 features 4.6 us (5.8 as one chain over K), K = 3,072 6.2 (14.9), 12,288 into 4,096 51 (81), 1,024 into
// 32,000 27 (4.9 TB/s). Eight rows, K = 3,072 into 1,024: 13.8 (24.8); 37 rows: 28 (46), 1,024 into 6,144 25 (47). KG = 1 (64 threads
// a block, several blocks an SM) for more than eight rows: with four segments in a block each SM's shared memory feeds four times
// the threads and fewer SMs have a block (37 rows, K = 1,024 into 1,024: 13 us, 23 before the blocks were made this small).
// ---------------------------------------------------------------------------------
template <typename TX, int RM, int TM, int CN, int TN, int KG, int BK, int NS, bool VEC>
__global__ void __launch_bounds__(RM * CN * KG)
gemm_f32_seg_kernel(const TX* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                    float* __restrict__ out, int M, int N, int K, long long x_stride, long long out_stride, int n_blocks) {
  constexpr int BM = RM * TM, BN = CN * TN, GT = RM * CN, THREADS = GT * KG, TILE = BM * BN;
  constexpr int XS = BK + 16 / (int)sizeof(TX), WS = BK + 4, STEPS = GF_SEG / BK;
  extern __shared__ __align__(16) unsigned char gf_raw[];
  float* part = reinterpret_cast<float*>(gf_raw);                 // [KG][TILE]
  float* total = part + KG * TILE;                                // [TILE]: of the rounds before, each element one thread's
  float* ws = total + TILE;                                       // [NS][KG][BN][WS]
  TX* xs = reinterpret_cast<TX*>(ws + NS * KG * BN * WS);         // [NS][KG][BM][XS]
  const int tid = threadIdx.x, g = tid / GT, tx = tid % GT % CN, ty = tid % GT / CN;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM, rank = blockIdx.z;      // n_blocks = the cluster's size = gridDim.z
  const int segments = (K + GF_SEG - 1) / GF_SEG, rounds = (segments + KG * n_blocks - 1) / (KG * n_blocks);
  const int steps = rounds * STEPS;
  pdl_launch_dependents();
  // Step `it` of round `it / STEPS`: BK values of each of the block's KG segments. A step that starts beyond K is neither filled nor read.
  auto k_of = [&](int it, int group) { return ((it / STEPS * n_blocks + rank) * KG + group) * GF_SEG + it % STEPS * BK; };
  // `rows` of each of the KG segments. Pieces of four values: those beyond the matrix are filled with zeros. Value by value a
  // thread's copies are many, so steps that start beyond K (which nothing reads) are left out.
  auto load = [&](auto* dst, const auto* src, long long src_stride, auto rows, int row0, int n_rows, int it) {
    using T = std::remove_reference_t<decltype(*dst)>;
    constexpr int ROWS = decltype(rows)::value, STRIDE = BK + 16 / (int)sizeof(T);
    dst += it % NS * (KG * ROWS * STRIDE);
    if constexpr (VEC) {
#pragma unroll
      for (int e = tid; e < KG * ROWS * (BK / 4); e += THREADS) {
        const int r = e / (BK / 4), c = e % (BK / 4) * 4, k = k_of(it, r / ROWS) + c, row = row0 + r % ROWS;
        const bool in = row < n_rows && k < K;
        const auto* from = in ? src + row * src_stride + k : src;
        if constexpr (sizeof(T) == 4) cp_async_16(dst + r * STRIDE + c, from, in ? 16 : 0);
        else cp_async_8(dst + r * STRIDE + c, from, in ? 8 : 0);
      }
    } else {
      constexpr int PASS = THREADS / BK;
      static_assert(THREADS % BK == 0, "whole rows a pass");
      const int c = tid % BK, k0 = k_of(it, 0);
      const int live = KG == 1 ? ROWS : min(KG, (K - k0 + GF_SEG - 1) / GF_SEG) * ROWS;
#pragma unroll
      for (int r0 = 0; r0 < KG * ROWS; r0 += PASS) {
        const int r = r0 + tid / BK;
        if (r >= live) break;
        const int k = k0 + r / ROWS * GF_SEG + c, row = row0 + r % ROWS;
        const bool in = row < n_rows && k < K;
        const auto* from = in ? src + row * src_stride + k : src;
        if constexpr (sizeof(T) == 4) cp_async_4(dst + r * STRIDE + c, from, in ? 4 : 0);
        else dst[r * STRIDE + c] = in ? *from : T(0.f);      // (no asynchronous copy has two bytes)
      }
    }
  };
  auto load_w = [&](int it) { load(ws, w, (long long)K, std::integral_constant<int, BN>{}, n0, N, it); };
  auto load_x = [&](int it) { load(xs, x, x_stride, std::integral_constant<int, BM>{}, m0, M, it); };
  // The weights of the first steps are on their way before the kernel that makes the rows has ended (steps >= NS - 1:
  // a round has GF_SEG / BK steps).
  static_assert(STEPS >= NS - 1, "the first stages lie in the first round");
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) load_w(s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < NS - 1; ++s) {
    load_x(s);
    cp_async_commit();      // (the first group holds the weights of all of them)
  }
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  const int share = (TILE + n_blocks - 1) / n_blocks, own_lo = rank * share, own_hi = min(TILE, own_lo + share);
  for (int it = 0; it < steps; ++it) {
    cp_async_wait<NS - 2>();
    __syncthreads();      // stage `it` is there for everyone, and everyone is done with the stage that is filled next
    if (it + NS - 1 < steps) {
      load_w(it + NS - 1);
      load_x(it + NS - 1);
    }
    cp_async_commit();
    const float* wr = ws + (it % NS * KG + g) * (BN * WS);
    const TX* xr = xs + (it % NS * KG + g) * (BM * XS);
    if (k_of(it, g) < K) {
      float4 av[2][TM], bv[2][TN];
      auto fetch = [&](int buf, int k0) {
#pragma unroll
        for (int i = 0; i < TM; ++i) av[buf][i] = gf_four(xr + (ty + i * RM) * XS + k0);
#pragma unroll
        for (int j = 0; j < TN; ++j) bv[buf][j] = gf_four(wr + (tx + j * CN) * WS + k0);
      };
      fetch(0, 0);
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        const int cur = (k / 4) & 1;
        if (k + 4 < BK) fetch(cur ^ 1, k + 4);
        gf_add<TM, TN>(acc, av[cur], bv[cur]);
      }
    }
    if (it % STEPS != STEPS - 1) continue;
    // The end of a round. (Segments beyond K leave zeros, which are not added.)
    if (it >= STEPS) gf_round_wait(n_blocks);      // everyone has read the sums of the round before
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        part[g * TILE + (ty + i * RM) * BN + tx + j * CN] = acc[i][j];
        acc[i][j] = 0.f;
      }
    gf_round_arrive(n_blocks);
    gf_round_wait(n_blocks);
    const int first = it / STEPS * n_blocks * KG, here = min(segments - first, n_blocks * KG);
    constexpr int AT_ONCE = 4;      // elements of a thread whose reads from a peer are in flight together
    for (int e0 = own_lo + tid; e0 < own_hi; e0 += AT_ONCE * THREADS) {
      float sum[AT_ONCE];
#pragma unroll
      for (int i = 0; i < AT_ONCE; ++i) sum[i] = it < STEPS || e0 + i * THREADS >= own_hi ? 0.f : total[e0 + i * THREADS];
      for (int s = 0; s < here; ++s) {
        const float* from = part + s % KG * TILE + e0;
        float v[AT_ONCE];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) v[i] = gf_peer(from + (e0 + i * THREADS < own_hi ? i * THREADS : 0), s / KG, n_blocks);
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) sum[i] += v[i];
      }
#pragma unroll
      for (int i = 0; i < AT_ONCE; ++i) {
        const int e = e0 + i * THREADS, m = m0 + e / BN, n = n0 + e % BN;
        if (e >= own_hi) continue;
        if (it + 1 < steps) total[e] = sum[i];
        else if (m < M && n < N) out[(size_t)m * out_stride + n] = sum[i] + (bias ? bias[n] : 0.f);
      }
    }
    gf_round_arrive(n_blocks);
  }
  gf_round_wait(n_blocks);      // no block leaves while its sums may be read
}


template <typename F, typename... Args>
static int gf_launch(F kernel, dim3 grid, int threads, size_t smem, bool pdl, cudaStream_t stream, Args... args) {
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return llmrs_fail("gemm_f32: shared memory %zu: %s", smem, cudaGetErrorString(e));
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (grid.z > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = grid.z;
  }
  if (pdl && g_llmrs_pdl) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cudaLaunchKernelEx(&cfg, kernel, args...);
  return llmrs_launch_status("gemm_f32");
}

template <typename TX>
struct GfArgs {
  const TX* x;
  long long x_stride;
  const float *w, *bias;
  float* out;
  long long out_stride;
  int M, N, K;
  bool vec;
  cudaStream_t stream;
};

template <int BM, int BN, int TM, int TN, int BK, int NS, bool IN_REGS, typename TX>
static int gf_tiles(const GfArgs<TX>& a) {
  constexpr int threads = (BM / TM) * (BN / TN);
  constexpr size_t smem = (IN_REGS ? 0 : (size_t)TM * TN * threads * 4) + (size_t)NS * (BN * (BK + 4) * 4 + BM * (BK * sizeof(TX) + 16));
  const dim3 grid((a.N + BN - 1) / BN, (a.M + BM - 1) / BM);
  LLMRS_REQUIRE(grid.y <= 65535, "gemm_f32: M=%d is too large", a.M);
  return gf_launch(a.vec ? gemm_f32_kernel<TX, BM, BN, TM, TN, BK, NS, true, IN_REGS> : gemm_f32_kernel<TX, BM, BN, TM, TN, BK, NS, false, IN_REGS>,
                   grid, threads, smem, false, a.stream, a.x, a.w, a.bias, a.out, a.M, a.N, a.K, a.x_stride, a.out_stride);
}

// Blocks a cluster where `cluster` is 0: as many as the device holds at a time (KG = 1: six an SM, of those that hold 32 rows), at most
// one for every KG segments, at most eight, and no more than leave the last round's blocks with segments (6,144 features of 16 rows,
// K = 1,024: four blocks 14.3 us, three, the last of which walk a second round alone, 25).
static long long gf_cluster(long long tiles, long long turns, int blocks) {
  const long long most = std::min(8ll, std::max(1ll, blocks / tiles)), rounds = (turns + most - 1) / most;
  return (turns + rounds - 1) / rounds;
}
template <typename TX>
constexpr size_t gf_seg_smem(int rows, int cols, int kg, int bk, int ns) {
  return (size_t)(kg + 1) * rows * cols * 4 + (size_t)ns * kg * (cols * (bk + 4) * 4 + rows * (bk * sizeof(TX) + 16));
}
template <int RM, int TM, int CN, int TN, int KG, int BK, int NS, typename TX>
static int gf_segments(const GfArgs<TX>& a, long long cluster = 0) {
  constexpr int BM = RM * TM, BN = CN * TN, threads = RM * CN * KG;
  constexpr size_t smem = gf_seg_smem<TX>(BM, BN, KG, BK, NS);
  static_assert(smem <= 227 * 1024, "the block's shared memory");
  const long long tiles_n = (a.N + BN - 1) / BN, tiles_m = (a.M + BM - 1) / BM;
  LLMRS_REQUIRE(tiles_m <= 65535, "gemm_f32: M=%d is too large", a.M);
  if (cluster == 0) cluster = gf_cluster(tiles_n * tiles_m, ((a.K + GF_SEG - 1) / GF_SEG + KG - 1) / KG, 148 * (KG > 1 ? 2 : 6));
  const dim3 grid((unsigned)tiles_n, (unsigned)tiles_m, (unsigned)cluster);
  return gf_launch(a.vec ? gemm_f32_seg_kernel<TX, RM, TM, CN, TN, KG, BK, NS, true>
                         : gemm_f32_seg_kernel<TX, RM, TM, CN, TN, KG, BK, NS, false>,
                   grid, threads, smem, true, a.stream, a.x, a.w, a.bias, a.out, a.M, a.N, a.K, a.x_stride, a.out_stride,
                   (int)cluster);
}

// Estimated us of tiles of `rows` x 32 by segments, clusters of so many blocks, to compare with one another. An SM's
// blocks share its path from shared memory, rows * (TM + TN) / (TM * TN) a segment; a block by itself waits for its own chain; blocks
// beyond those that an SM holds wait for a wave. Fitted to 149 products (65 to 576 rows, 512 to 3,072 features, K 768 to 3,072), all
// tiles and clusters beside one another: the choice below takes 1.05 times as long as the best one on average, 1.28 at worst;
// by the empty rows alone it was 1.14 and 1.86 (408 rows, K = 1,024 into 1,024: 57 us in tiles of 24, 41 so).
template <typename TX>
static double gf_seg_us(int rows, long long cluster, long long M, long long N, long long K) {
  const long long turns = (K + GF_SEG - 1) / GF_SEG;
  const double work = rows * (rows / 8 + 4.0) / (rows / 8 * 4);
  const long long resident = (227 * 1024) / (long long)(gf_seg_smem<TX>(rows, 32, 1, 32, 3) + 1024);
  const long long blocks = ((M + rows - 1) / rows) * ((N + 31) / 32) * cluster, waves = blocks / (148 * resident), rest = blocks - waves * 148 * resident;
  auto segment = [&](double an_sm) { return std::max(2.548 + 0.21 * work, 0.075 * work * an_sm); };
  const double at_once = waves * segment(resident) + (rest ? segment((rest + 147) / 148) : 0.0);
  return (turns + cluster - 1) / cluster * (at_once + 3.744) + 1.54 * (waves + (rest ? 1 : 0));
}

// Many rows: the largest tile of which there are enough blocks for the SMs, since larger tiles read the operands less often.
// Otherwise segments side by side. Both sides of the lines, measured: 48 rows of 1,024 into 6,144 features 31 us by segments,
// 47 in tiles of 64 x 64; 90 rows 59 in tiles of 48 rows by segments, 76 in 192 tiles of 64 x 64, but 300 rows 144 so and 148;
// 16 rows of tiles of eight features (K = 1,024 into 2,048) 12.1 us, 2,048 features of one row 5.0 in tiles of eight, 7.0 in tiles of 32.
template <typename TX>
static int gemm_f32_any(const TX* x, long long x_stride, const float* w, const float* bias, float* out,
                        long long out_stride, int M, int N, int K, cudaStream_t stream) {
  LLMRS_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
  if (M == 0) return 0;
  // Pieces of four values by one asynchronous copy each: every row of both operands must start on such a piece.
  const bool vec = K % 4 == 0 && x_stride % 4 == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)x & (4 * sizeof(TX) - 1)) == 0;
  const GfArgs<TX> a{x, x_stride, w, bias, out, out_stride, M, N, K, vec, stream};
  auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  constexpr int ENOUGH = 148;
  if (M > 64 && blocks(128, 128) >= ENOUGH) {
    if (!vec) return gf_tiles<128, 128, 8, 8, 32, 4, true>(a);
    return gf_tiles<128, 128, 8, 8, 32, sizeof(TX) == 4 ? 3 : 4, false>(a);
  }
  if (M > 48 && blocks(64, 64) >= ENOUGH) return gf_tiles<64, 64, 4, 8, 32, 4, true>(a);
  const bool narrow = N <= 16 * ENOUGH;      // tiles of eight features: twice as many as SMs at most
  if (M == 1) return narrow ? gf_segments<1, 1, 8, 1, 16, 32, 4>(a) : gf_segments<1, 1, 32, 1, 4, 32, 4>(a);
  if (M <= 4) return narrow ? gf_segments<1, 4, 8, 1, 16, 32, 3>(a) : gf_segments<1, 4, 32, 1, 4, 32, 4>(a);
  if (M <= 8) return narrow ? gf_segments<1, 8, 8, 1, 16, 32, 3>(a) : gf_segments<1, 8, 32, 1, 4, 32, 4>(a);
  if (M <= 16) return gf_segments<4, 4, 8, 4, 1, 32, 3>(a);
  // (Value by value a block of 128 threads gets its copies out sooner: 300 rows of 1,023 into 1,500 features 54 us, 75 by segments.)
  if (!vec && M > 64) return gf_tiles<32, 32, 2, 4, 32, 4, true>(a);
  int rows = 0;      // of a tile: those that leave the fewest empty, of equals the most
  for (int r : {64, 48, 40, 32, 24})
    if (rows == 0 || blocks(r, N) * r < blocks(rows, N) * rows) rows = r;
  long long cluster = 0;
  if (M > 64) {      // several tiles of rows: waves weigh more than empty rows do; another choice has to promise an eighth
    const long long turns = (K + GF_SEG - 1) / GF_SEG;
    cluster = gf_cluster(blocks(rows, 32), turns, 148 * 6);
    double best = 0.87 * gf_seg_us<TX>(rows, cluster, M, N, K);
    for (int r : {24, 32, 40, 48, 64})
      for (long long c : {1, 2, 3, 4, 6, 8}) {
        const long long rounds = (turns + c - 1) / c;
        if (c > turns || (turns + rounds - 1) / rounds != c) continue;
        const double us = gf_seg_us<TX>(r, c, M, N, K);
        if (us < best) best = us, rows = r, cluster = c;
      }
  }
  switch (rows) {
    case 24: return gf_segments<8, 3, 8, 4, 1, 32, 3>(a, cluster);
    case 32: return gf_segments<8, 4, 8, 4, 1, 32, 3>(a, cluster);
    case 40: return gf_segments<8, 5, 8, 4, 1, 32, 3>(a, cluster);
    case 48: return gf_segments<8, 6, 8, 4, 1, 32, 3>(a, cluster);
    default: return gf_segments<8, 8, 8, 4, 1, 32, 3>(a, cluster);
  }
}

LLMRS_API int llmrs_gemm_f32(const float* x, long long x_stride, const float* w, const float* bias, float* out,
                             long long out_stride, int M, int N, int K, cudaStream_t stream) {
  return gemm_f32_any<float>(x, x_stride, w, bias, out, out_stride, M, N, K, stream);
}

// The same product for rows stored in bfloat16 (activations of the bfloat16 path whose product must not be rounded:
// a router's logits, the gates of a recurrence): the rows are widened as they are read, weights, sums and output
// are float32.
LLMRS_API int llmrs_gemm_f32_bf16_rows(const void* x, long long x_stride, const float* w, const float* bias, float* out,
                                       long long out_stride, int M, int N, int K, cudaStream_t stream) {
  return gemm_f32_any<__nv_bfloat16>((const __nv_bfloat16*)x, x_stride, w, bias, out, out_stride, M, N, K, stream);
}

// ---------------------------------------------------------------------------------
// Few output features (a router's logits, the gates of a recurrence, a single gate row): out[m, n] for n < N <= some
// hundreds. The tiled kernel above would run as one or two blocks that walk K alone; here a block holds SK_TOKENS
// rows of x in shared memory and each of its warps owns one output feature: its lanes walk that weight row once,
// four values per load, against all the block's rows. Every output is summed in the same order whatever M is (a
// lane's own values in order of k, then the lanes by butterfly), so a token's result does not depend on the batch.
// ---------------------------------------------------------------------------------
constexpr int SK_WARPS = 8, SK_THREADS = SK_WARPS * 32, SK_TOKENS = 8;

// SPLIT false: a warp owns a feature and walks all of K. SPLIT true (few rows: decoding): a block owns ONE feature,
// its warps walk an eighth of K each and the block adds the eight parts in warp order, so that a product of a
// handful of rows still fills the device.
template <typename TX, bool SPLIT>
__global__ void __launch_bounds__(SK_THREADS)
gemm_f32_skinny_kernel(const TX* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       float* __restrict__ out, int M, int N, int K, long long x_stride, long long out_stride) {
  extern __shared__ __align__(16) unsigned char sk_raw[];
  __shared__ float parts[SK_WARPS][SK_TOKENS];
  TX* xs = reinterpret_cast<TX*>(sk_raw);      // [SK_TOKENS][K]
  const int m0 = blockIdx.x * SK_TOKENS, rows = min(SK_TOKENS, M - m0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  static_assert(SK_WARPS == SK_TOKENS, "a warp a row");
  // Sixteen bytes at a time, a warp a row, where rows start on such a boundary (value by value with a division each, the rows took
  // longer than the product: 8 bfloat16 rows of 2,048 into 33 features 9.1 us, 3.7 so).
  constexpr int PIECE = 16 / (int)sizeof(TX);
  if (K % PIECE == 0 && x_stride % PIECE == 0 && ((uintptr_t)x & 15) == 0) {
    const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)(m0 + min(warp, rows - 1)) * x_stride);
    uint4* to = reinterpret_cast<uint4*>(xs + (size_t)warp * K);
#pragma unroll 4
    for (int i = lane; i < K / PIECE; i += 32) to[i] = warp < rows ? __ldg(from + i) : make_uint4(0u, 0u, 0u, 0u);
  } else {
    for (int i = threadIdx.x; i < SK_TOKENS * K; i += SK_THREADS) {
      const int r = i / K, k = i - r * K;
      xs[i] = r < rows ? x[(size_t)(m0 + r) * x_stride + k] : TX(0.f);
    }
  }
  __syncthreads();
  const int n = SPLIT ? (int)blockIdx.y : (int)blockIdx.y * SK_WARPS + warp;
  const bool live = n < N;
  const float* wr = w + (size_t)(live ? n : 0) * K;
  float acc[SK_TOKENS];
#pragma unroll
  for (int r = 0; r < SK_TOKENS; ++r) acc[r] = 0.f;
  const int K4 = K & ~3;
  // The piece of K this warp walks: all of it, or its eighth (in whole groups of 128).
  const int piece = SPLIT ? (((K4 + 127) / 128 + SK_WARPS - 1) / SK_WARPS) * 128 : K4;
  const int k_lo = SPLIT ? warp * piece : 0, k_hi = min(K4, k_lo + piece);
  if (live) {
    for (int k = k_lo + lane * 4; k < k_hi; k += 128) {
      const float4 wv = __ldg(reinterpret_cast<const float4*>(wr + k));
#pragma unroll
      for (int r = 0; r < SK_TOKENS; ++r) {
        const float4 xv = gf_four(xs + r * K + k);      // (K is a multiple of four)
        acc[r] = fmaf(xv.x, wv.x, acc[r]);
        acc[r] = fmaf(xv.y, wv.y, acc[r]);
        acc[r] = fmaf(xv.z, wv.z, acc[r]);
        acc[r] = fmaf(xv.w, wv.w, acc[r]);
      }
    }
    if (!SPLIT || warp == SK_WARPS - 1)
      for (int k = K4 + lane; k < K; k += 32) {
#pragma unroll
        for (int r = 0; r < SK_TOKENS; ++r) acc[r] = fmaf(to_float(xs[r * K + k]), wr[k], acc[r]);
      }
  }
#pragma unroll
  for (int r = 0; r < SK_TOKENS; ++r) {
    const float s = warp_sum(acc[r]);
    if (SPLIT) {
      if (lane == 0) parts[warp][r] = s;
    } else if (lane == 0 && live && r < rows) {
      out[(size_t)(m0 + r) * out_stride + n] = s + (bias ? bias[n] : 0.f);
    }
  }
  if (SPLIT) {
    __syncthreads();
    if (threadIdx.x < rows && live) {
      float s = 0.f;
#pragma unroll
      for (int wv = 0; wv < SK_WARPS; ++wv) s += parts[wv][threadIdx.x];
      out[(size_t)(m0 + threadIdx.x) * out_stride + n] = s + (bias ? bias[n] : 0.f);
    }
  }
}

// x_dtype: LLMRS_F32 or LLMRS_BF16 rows; w (16-byte aligned rows: K % 4 == 0), bias and out float32.
LLMRS_API int llmrs_gemm_f32_skinny(const void* x, int x_dtype, long long x_stride, const float* w, const float* bias,
                                    float* out, long long out_stride, int M, int N, int K, cudaStream_t stream) {
  LLMRS_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_skinny: bad sizes M=%d N=%d K=%d", M, N, K);
  LLMRS_REQUIRE(((uintptr_t)w & 15) == 0, "gemm_f32_skinny: the weights must be 16-byte aligned");
  if (M == 0) return 0;
  const size_t smem = (size_t)SK_TOKENS * K * (x_dtype == LLMRS_F32 ? 4 : 2);
  LLMRS_REQUIRE(smem <= 200 * 1024, "gemm_f32_skinny: rows of %d values are too long", K);
  // (48 KB need no asking, but the kernel's own `parts` counts too: eight rows of 1,536 floats are 48 KB by themselves.)
  const bool split = M <= 4 * SK_TOKENS;       // few rows: a block per feature
  dim3 grid((M + SK_TOKENS - 1) / SK_TOKENS, split ? N : (N + SK_WARPS - 1) / SK_WARPS);
  LLMRS_REQUIRE(grid.y <= 65535, "gemm_f32_skinny: N=%d is too large", N);
#define LLMRS_SK_LAUNCH(T, S)                                                                                         \
  do {                                                                                                                \
    static size_t configured = 40 * 1024;                                                                             \
    if (smem > configured) {                                                                                          \
      cudaError_t e = cudaFuncSetAttribute(gemm_f32_skinny_kernel<T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                           (int)smem);                                                                \
      if (e != cudaSuccess) return llmrs_fail("gemm_f32_skinny: shared memory %zu: %s", smem, cudaGetErrorString(e)); \
      configured = smem;                                                                                              \
    }                                                                                                                 \
    gemm_f32_skinny_kernel<T, S><<<grid, SK_THREADS, smem, stream>>>((const T*)x, w, bias, out, M, N, K, x_stride,    \
                                                                     out_stride);                                     \
  } while (0)
  if (x_dtype == LLMRS_F32 && split) LLMRS_SK_LAUNCH(float, true);
  else if (x_dtype == LLMRS_F32) LLMRS_SK_LAUNCH(float, false);
  else if (x_dtype == LLMRS_BF16 && split) LLMRS_SK_LAUNCH(__nv_bfloat16, true);
  else if (x_dtype == LLMRS_BF16) LLMRS_SK_LAUNCH(__nv_bfloat16, false);
  else return llmrs_fail("gemm_f32_skinny: unknown dtype %d", x_dtype);
#undef LLMRS_SK_LAUNCH
  return llmrs_launch_status("gemm_f32_skinny");
}
