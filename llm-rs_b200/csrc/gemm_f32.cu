// True 32-bit matrix product for the float32 path: out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]).
//
// FFMA on the CUDA cores, no tensor-core mode of reduced precision. Every output
// element is summed over k in the same order whatever M is, so a token's result does
// not depend on what else is in the batch. The reference's products are library calls
// (llm-core/src/backends/candle.rs:1276-1340: weight [out, in], used transposed,
// optional bias added after).
#include "common.cuh"
#include "mma_util.cuh"

// A block owns a tile of BM rows x BN features and walks K in steps of BK through NS stages of shared memory, filled by
// asynchronous copies NS - 1 steps ahead. Both operands stay in rows along K as they come, a row padded by 16 bytes so that
// neighbouring rows' 16-byte reads fall into different banks; a thread reads four values of K of its TM rows and TN
// features at a time and adds them in order of K. An output is ONE chain of fused multiply-adds whatever the tile, which
// keeps its bits the same in every batch, and is why no tile splits K: a product of few rows is bound by that chain and by
// the latency of its stages (K = 3,072 into 1,024 features, one row: 15.5 us, 236 before with one synchronous stage of 16
// values), one of many features by the stream of its weights (1,024 into 32,000: 35 us, 3.7 TB/s; 185 before), one of many
// rows by the FMA units (2,048 rows of 4,096 x 4,096: 1,867 us, 36.8 TFLOP/s; 2,711 before).
// (A tile of few outputs has more threads than outputs: its copies are dealt out over four warps, so that the one that adds loses
// less time to them.)
__host__ __device__ constexpr int gf_threads(int bm, int bn, int tm, int tn) {
  return (bm / tm) * (bn / tn) < 128 ? 128 : (bm / tm) * (bn / tn);
}
template <typename TX, int BM, int BN, int TM, int TN, int BK, int NS, int U, bool VEC>
__global__ void __launch_bounds__(gf_threads(BM, BN, TM, TN))
gemm_f32_kernel(const TX* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ out, int M, int N, int K, long long x_stride, long long out_stride) {
  constexpr int THREADS = gf_threads(BM, BN, TM, TN), CN = BN / TN, RM = BM / TM;
  constexpr int XS = BK + 16 / (int)sizeof(TX), WS = BK + 4;      // elements a row of a stage takes
  extern __shared__ __align__(16) unsigned char gf_raw[];
  float* ws = reinterpret_cast<float*>(gf_raw);                   // [NS][BN][WS]
  TX* xs = reinterpret_cast<TX*>(gf_raw + sizeof(float) * NS * BN * WS);      // [NS][BM][XS]
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
      // Value by value: a thread keeps to a column (to every THREADS-th of a wide step) and goes down the rows, so that an address
      // is one addition (1,000 rows of 1,023 into 1,024 features 72 us; 141 with an address and plain loads a value, 94 by the
      // kernel before; 2,050 into 2,048 276, 523 and 367).
      constexpr int COLS = BK < THREADS ? BK : THREADS, PASS = THREADS / COLS;
#pragma unroll
      for (int c0 = 0; c0 < BK; c0 += COLS) {
        const int c = c0 + tid % COLS, r0 = tid / COLS;
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
    }
    cp_async_commit();
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
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
    if (RM * CN < THREADS && tid >= RM * CN) continue;      // only copies
    const float* wr = ws + (it % NS) * BN * WS;
    const TX* xr = xs + (it % NS) * BM * XS;
    // The next U pieces are read while the present ones are added: a warp alone on its scheduler would otherwise wait
    // for shared memory in every step of its chains.
    float4 av[2][U][TM], bv[2][U][TN];
    auto fetch = [&](int buf, int k0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const TX* p = xr + (ty + i * RM) * XS + k0 + 4 * u;
          if constexpr (sizeof(TX) == 4) {
            av[buf][u][i] = *reinterpret_cast<const float4*>(p);
          } else {
            const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
            const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + 2));
            av[buf][u][i] = make_float4(lo.x, lo.y, hi.x, hi.y);
          }
        }
#pragma unroll
        for (int j = 0; j < TN; ++j)
          bv[buf][u][j] = *reinterpret_cast<const float4*>(wr + (tx + j * CN) * WS + k0 + 4 * u);
      }
    };
    fetch(0, 0);
#pragma unroll
    for (int k = 0; k < BK; k += 4 * U) {
      const int cur = (k / (4 * U)) & 1;
      if (k + 4 * U < BK) fetch(cur ^ 1, k + 4 * U);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const float4 a = av[cur][u][i], b = bv[cur][u][j];
            acc[i][j] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc[i][j]))));
          }
    }
  }
  if (RM * CN < THREADS && tid >= RM * CN) return;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * RM;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * CN;
      if (n < N) out[(size_t)m * out_stride + n] = acc[i][j] + (bias ? bias[n] : 0.f);
    }
  }
}

template <typename TX, int BM, int BN, int TM, int TN, int BK, int NS, int U>
static int launch_gemm_f32(bool vec, const TX* x, long long x_stride, const float* w, const float* bias, float* out,
                           long long out_stride, int M, int N, int K, cudaStream_t stream) {
  constexpr size_t smem = (size_t)NS * (BN * (BK + 4) * sizeof(float) + BM * (BK * sizeof(TX) + 16));
  constexpr int threads = gf_threads(BM, BN, TM, TN);
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  LLMRS_REQUIRE(grid.y <= 65535, "gemm_f32: M=%d is too large", M);
  auto go = [&](auto kernel) {
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return llmrs_fail("gemm_f32: shared memory %zu: %s", smem, cudaGetErrorString(e));
    }
    kernel<<<grid, threads, smem, stream>>>(x, w, bias, out, M, N, K, x_stride, out_stride);
    return llmrs_launch_status("gemm_f32");
  };
  return vec ? go(gemm_f32_kernel<TX, BM, BN, TM, TN, BK, NS, U, true>) : go(gemm_f32_kernel<TX, BM, BN, TM, TN, BK, NS, U, false>);
}

// The largest tile of which there are enough blocks for the SMs: larger tiles read the operands less often, smaller ones
// spread a short product over the device, and no tile has more rows than the product would half fill. Both sides of the
// line, measured: 16 rows of 2,048 into 6,144 features 43 us in tiles of 16 x 32, 72 in tiles of 32 x 32 whose second half
// is empty; 37 rows of 1,024 into 6,144 features 48 us in 384 tiles of 32 x 32, 80 in 96 tiles of 64 x 64 (as before).
template <typename TX>
static int gemm_f32_any(const TX* x, long long x_stride, const float* w, const float* bias, float* out,
                        long long out_stride, int M, int N, int K, cudaStream_t stream) {
  LLMRS_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
  if (M == 0) return 0;
  // Pieces of four values by one asynchronous copy each: every row of both operands must start on such a piece.
  const bool vec = K % 4 == 0 && x_stride % 4 == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)x & (4 * sizeof(TX) - 1)) == 0;
  auto blocks = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  constexpr int ENOUGH = 148;
#define LLMRS_GF(BM, BN, TM, TN, BK, NS, U) \
  return launch_gemm_f32<TX, BM, BN, TM, TN, BK, NS, U>(vec, x, x_stride, w, bias, out, out_stride, M, N, K, stream)
  if (M > 64 && blocks(128, 128) >= ENOUGH) LLMRS_GF(128, 128, 8, 8, 16, 4, 1);
  if (M > 32 && blocks(64, 64) >= ENOUGH) LLMRS_GF(64, 64, 4, 8, 32, 4, 1);
  if (M > 16 && blocks(32, 32) >= ENOUGH) LLMRS_GF(32, 32, 2, 4, 32, 4, 1);
  if (M > 8 && blocks(16, 32) >= ENOUGH) LLMRS_GF(16, 32, 2, 2, 64, 4, 2);
  if (M > 4 && blocks(8, 32) >= ENOUGH) LLMRS_GF(8, 32, 2, 1, 64, 4, 4);
  if (M > 4) LLMRS_GF(8, 16, 1, 1, 64, 4, 4);
  if (M == 1) {      // tiles of one row read the weights from shared memory once, where those of four rows read them for each: 1,024
                     // into 32,000 features 35 us (46), into 6,144 9.8 (14), K = 3,072 into 1,024 15.5 (19)
    if (N >= 64 * 2 * ENOUGH) LLMRS_GF(1, 64, 1, 1, 64, 3, 4);
    if (N >= 32 * ENOUGH) LLMRS_GF(1, 32, 1, 1, 128, 4, 4);
    if (N >= 16 * ENOUGH) LLMRS_GF(1, 16, 1, 1, 128, 6, 4);
    LLMRS_GF(1, 8, 1, 1, 256, 6, 4);
  }
  if (blocks(4, 32) >= 2 * ENOUGH) LLMRS_GF(4, 32, 1, 1, 64, 4, 4);
  LLMRS_GF(4, 8, 1, 1, 128, 4, 4);
#undef LLMRS_GF
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
  for (int i = threadIdx.x; i < SK_TOKENS * K; i += SK_THREADS) {
    const int r = i / K, k = i - r * K;
    xs[i] = r < rows ? x[(size_t)(m0 + r) * x_stride + k] : TX(0.f);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
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
      const float4 wv = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
      for (int r = 0; r < SK_TOKENS; ++r) {
        const TX* xr = xs + r * K + k;
        acc[r] = fmaf(to_float(xr[0]), wv.x, acc[r]);
        acc[r] = fmaf(to_float(xr[1]), wv.y, acc[r]);
        acc[r] = fmaf(to_float(xr[2]), wv.z, acc[r]);
        acc[r] = fmaf(to_float(xr[3]), wv.w, acc[r]);
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
