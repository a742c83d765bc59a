// The walk of a request's tokens that the recurrences with a matrix state S [key channel, value channel] share, four
// tokens a turn, for the heads that the chunks of sixteen tokens on the tensor cores (state_chunks.cuh) do not take: a number of
// channels that four does not divide, or more than 128 key channels (64 under the generalized rule). With S_0 the state before a turn and i, j the turn's tokens:
//
//   WALK_LINEAR    y_i = gain_i v_i                                         o_i = P_i (q_i . S_0) + sum_{j<=i} Q_ij y_j
//   WALK_GATED     y_i = beta_i (v_i - P_i (k_i . S_0) - sum_{j<i} K_ij y_j)        the same o_i
//                  S_4 = P_4 S_0 + sum_j (Z_j k_j) y_j            (a decay per token: P_i up to and with i, Z_j after j)
//   WALK_CHANNEL   the same with a decay per key channel, which then lies in the rows: q_i, k_i decayed from the turn's
//                  start up to and with i for the products with S_0, k_j decayed from j to the turn's end for the write
//   WALK_GENERAL   x_i = u_i . S_0 + sum_{j<i} (B_ij v_j + A_ij x_j),       o_i = r_i . S_0 + sum_{j<=i} (R_ij v_j + Q_ij x_j)
//                  S_4 = W S_0 + sum_j k_j v_j^T + a_j x_j^T      (rows decayed likewise, a_j the removal with its sign)
//
// The coefficients between two tokens of a turn (K, Q, A, B, R: products of two rows with the decays between them) do not
// depend on the state: they are made for all turns at once, ahead of the walk. What that buys: the products of all four
// tokens' rows with S_0 are independent of one another, so the sums over the lanes that share a column run side by side,
// where a walk token by token waits for one such chain in every token. Everything is float32; sums are in a fixed order.
//
// A block takes 16 value columns of a head with four warps. Sixteen neighbouring lanes share two columns; lane p of them
// holds key channels 4 (p + 16 j) .. + 3 of both. What bounds the walk is the path from shared memory to registers, 128
// bytes a cycle whatever lanes read the same address: a row's values are read once for two columns (with a column a lane,
// half of that path was busy with rows alone and 2,048 tokens took 276 us), while more columns a lane cost more shuffles
// than they save reads. Products run as packed pairs of float32 along the channels. The eight sums of a turn (four tokens,
// two columns) are dealt out over the lanes as they are summed: eight shuffles instead of the 32 of eight full sums. Rows
// arrive by 16-byte asynchronous copies through a ring of four stages of two turns, which are one stretch of code: a turn's
// read-outs are summed under the next one's products. What later tokens of the turn write is masked out of a token's read-out
// bit by bit: a coefficient of zero would not do, zero times an infinite value is no number. (Gated 402 us without, 406 with it;
// selects or branches in its place
// broke the stretch up: 437 and 485.)
//
// Measured against the walk token by token (one by one -> in turns, the recurrence alone, bfloat16 models): gated, 2,048 tokens
// of 16 heads of 128 x 128: 497 -> 265 us; general, 32 heads of 64 x 64: 816 -> 246 us; linear with a normaliser, portions of
// 1,311, 402 and 77 tokens beside single ones, 16 heads of 128 x 128: 496 -> 200 us. Now bound by issue: a warp alone on its
// scheduler (128 blocks on 148 SMs) gets an instruction out every second cycle at best and needs 90 a token.
#pragma once
#include "common.cuh"
#include "mma_util.cuh"

enum { WALK_LINEAR = 0, WALK_GATED = 1, WALK_CHANNEL = 2, WALK_GENERAL = 3 };
constexpr int WALK_TURN = 4, WALK_COLS = 16, WALK_LANES = 16, WALK_THREADS = WALK_COLS / 2 * WALK_LANES;
constexpr int WALK_STAGE = 2 * WALK_TURN, WALK_STAGES = 4;      // tokens of a stage, stages
// Which requests of a step are walked in turns is the caller's choice, by their tokens (`from`; see ops.walk_from): the kernels
// here leave shorter requests alone, the ones that walk token by token leave the others. Measured, token by token against in
// turns with its coefficients (us, one portion, the two kernels alone): 32 tokens gated 10.8 / 13.7, linear 11.5 / 12.8, general
// 18.3 / 19.6; 48 tokens 14.6 / 15.9, 15.6 / 14.4, 24.2 / 21.4; 64 tokens 18.5 / 17.8, 19.6 / 16.0, 30.7 / 23.4.

// A turn's coefficients of one head, in floats. LINEAR, GATED, CHANNEL: P [4] (CHANNEL: ones), Z [4] (likewise), beta or gain
// [4], K below the diagonal row by row [6] and two zeros, Q [4][4] (zero above the diagonal). GENERAL: A [6] + 2, B [6] + 2,
// R [4][4], Q [4][4].
constexpr int WALK_P = 0, WALK_Z = 4, WALK_BETA = 8, WALK_K = 12, WALK_Q = 20;
constexpr int WALK_GA = 0, WALK_GB = 8, WALK_GR = 16, WALK_GQ = 32;
__host__ __device__ constexpr int walk_table(int mode) { return mode == WALK_GENERAL ? 48 : 36; }
// The place of a request's first turn among all turns: requests' turns follow one another, floor(q_start / 4) + request
// leaves every request at least ceil(n / 4) places.
__host__ __device__ inline int walk_place(int q_start, int req) { return q_start / WALK_TURN + req; }
inline long long walk_places(int n_tokens, int n_requests) { return (long long)n_tokens / WALK_TURN + n_requests + 1; }
// The request whose turns place p lies among (the last one that starts at or before it); all lanes of a warp call it.
__device__ __forceinline__ int walk_request(const int* __restrict__ q_start, int n_requests, int p) {
  int found = 0;
  for (int base = 0; base < n_requests; base += 32) {
    const int r = base + (threadIdx.x & 31);
    const unsigned hit = __ballot_sync(0xffffffffu, r < n_requests && walk_place(q_start[r], r) <= p);
    if (hit == 0) break;
    found = base + 31 - __clz(hit);
  }
  return found;
}

// The request that token t belongs to; all lanes of a warp call it.
__device__ __forceinline__ int walk_token_request(const int* __restrict__ q_start, int n_requests, int t) {
  int found = 0;
  for (int base = 0; base < n_requests; base += 32) {
    const int r = base + (threadIdx.x & 31);
    const unsigned hit = __ballot_sync(0xffffffffu, r < n_requests && q_start[r] <= t);
    if (hit == 0) break;
    found = base + 31 - __clz(hit);
  }
  return found;
}

// Packed pairs of float32 in one 64-bit register.
typedef unsigned long long f2;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float f2_sum(f2 v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ float walk_keep(float v, unsigned mask) { return __uint_as_float(__float_as_uint(v) & mask); }

// Sums eight values over sixteen neighbouring lanes: lanes p and p + 8 end with the sum of value p & 7.
__device__ __forceinline__ float walk_sum8(const float (&v)[8], int part) {
  float a[4], b[2];
  const bool b2 = part & 4, b1 = part & 2, b0 = part & 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = (b2 ? v[4 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, b2 ? v[i] : v[4 + i], 4);
#pragma unroll
  for (int i = 0; i < 2; ++i) b[i] = (b1 ? a[2 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, b1 ? a[i] : a[2 + i], 2);
  const float c = (b0 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, b0 ? b[0] : b[1], 1);
  return c + __shfl_xor_sync(0xffffffffu, c, 8);
}
// Sums N values (16 or 32) over a warp: lane l ends with the sum of value l % N.
template <int N>
__device__ __forceinline__ float walk_sum_all(float (&v)[N], int lane) {
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1) {
    const bool hi = lane & half;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = hi ? v[half + i] : v[i], give = hi ? v[i] : v[half + i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
    }
  }
  return N == 16 ? v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16) : v[0];
}

// A row's channels as a warp holds them: lane l has channels V l .. V l + V - 1 of every 32 V, V = 4 (2 with two channels a
// lane). vec: rows start on boundaries of V values and d is a multiple of V. Channels >= d, and rows that are not there,
// are zero.
template <int CPL, typename T>
__device__ __forceinline__ void walk_load(const T* row, int lane, int d, bool there, bool vec, float (&out)[CPL]) {
  constexpr int V = CPL < 4 ? CPL : 4;
  struct alignas(V * sizeof(T)) Piece { T x[V]; };
#pragma unroll
  for (int m = 0; m < CPL; m += V) {
    const int c = V * lane + 32 * m;
    if (vec) {
      Piece in;
      if (there && c < d) in = *reinterpret_cast<const Piece*>(row + c);
#pragma unroll
      for (int e = 0; e < V; ++e) out[m + e] = there && c < d ? to_float(in.x[e]) : 0.f;
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e) out[m + e] = there && c + e < d ? to_float(row[c + e]) : 0.f;
    }
  }
}
template <int CPL>
__device__ __forceinline__ void walk_store(float* row, int lane, int d, bool vec, const float (&x)[CPL]) {
  constexpr int V = CPL < 4 ? CPL : 4;
  struct alignas(V * sizeof(float)) Piece { float x[V]; };
#pragma unroll
  for (int m = 0; m < CPL; m += V) {
    const int c = V * lane + 32 * m;
    if (vec && c < d) {
      Piece out;
#pragma unroll
      for (int e = 0; e < V; ++e) out.x[e] = x[m + e];
      *reinterpret_cast<Piece*>(row + c) = out;
    } else if (!vec) {
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (c + e < d) row[c + e] = x[m + e];
    }
  }
}

struct WalkArgs {
  // Row planes, each [tokens, stride] with head h's channels at (h / (heads / groups)) * d: the rows multiplied with S_0 (q;
  // k, u), the rows written (k, a) and the decay of a whole turn per channel [places, heads * d].
  const float *q, *k, *kb, *ab, *w;
  long long q_stride, k_stride, b_stride;
  const float* v;              // [tokens, heads * dv]
  const float* tables;         // [places, heads, walk_table]
  const float* skip;           // per head or null: o += skip * v
  float* state;                // [slots, heads, d, dv]
  float* norm_state;           // [slots, heads, d] or null: one more column whose value is 1
  float *o_raw, *nq;           // [tokens, heads * dv], [tokens, heads]
  const int *q_start, *n_new, *slot_ids;
  int n_heads, n_groups, d, dv;
  int from;                    // requests of fewer tokens are not walked here
};

// Rows a token brings in a stage.
__host__ __device__ constexpr int walk_rows(int mode) { return mode == WALK_GENERAL ? 4 : (mode == WALK_CHANNEL ? 3 : 2); }
__host__ __device__ constexpr bool walk_channel_decay(int mode) { return mode == WALK_CHANNEL || mode == WALK_GENERAL; }
__host__ __device__ constexpr int walk_stage_floats(int mode, int dmax) {
  return walk_rows(mode) * WALK_STAGE * dmax + (walk_channel_decay(mode) ? 2 * dmax : 0) + WALK_STAGE * WALK_COLS +
         2 * walk_table(mode);
}

// SOME: only requests of at least p.from tokens. (A template: the test alone changed the schedule of the gated walk from 266 to
// 275 us.)
template <int MODE, int DMAX, bool SOME>
__global__ void __launch_bounds__(WALK_THREADS, 2) state_walk_kernel(WalkArgs p, int col_blocks) {
  constexpr int IPL = DMAX / WALK_LANES, PAIRS = IPL / 2, ROWS = walk_rows(MODE), TAB = walk_table(MODE);
  constexpr bool CHANNEL = walk_channel_decay(MODE), KEEP = MODE == WALK_GATED && DMAX <= 128;
  constexpr int STAGE = walk_stage_floats(MODE, DMAX);
  constexpr int AT_W = ROWS * WALK_STAGE * DMAX, AT_V = AT_W + (CHANNEL ? 2 * DMAX : 0), AT_T = AT_V + WALK_STAGE * WALK_COLS;
  extern __shared__ __align__(16) float walk_smem[];
  // A request's blocks follow one another: the blocks of a long portion then start together, an SM each.
  const int req = blockIdx.x / (col_blocks * p.n_heads), head = blockIdx.x / col_blocks % p.n_heads;
  const int col0 = blockIdx.x % col_blocks * WALK_COLS, tid = threadIdx.x;
  const int part = tid % WALK_LANES, c0 = tid / WALK_LANES * 2, col = col0 + c0;      // this thread's columns: col, col + 1
  const int n = p.n_new[req], t0 = p.q_start[req], d = p.d, dv = p.dv, kh = head / (p.n_heads / p.n_groups);
  if (n <= 0 || (SOME && n < p.from)) return;
  const size_t slot = (size_t)p.slot_ids[req];
  float* S_g = p.state + (slot * p.n_heads + head) * (size_t)d * dv;
  float* N_g = p.norm_state ? p.norm_state + (slot * p.n_heads + head) * (size_t)d : nullptr;
  const bool norm[2] = {N_g != nullptr && col == dv, N_g != nullptr && col + 1 == dv};
  const bool live[2] = {col < dv || norm[0], col + 1 < dv || norm[1]};
  auto channel = [&](int i) { return ((i >> 2) * WALK_LANES + part) * 4 + (i & 3); };
  auto state_at = [&](int i, int c) { return norm[c] ? N_g + channel(i) : S_g + (size_t)channel(i) * dv + col + c; };
  f2 S[2][PAIRS];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int m = 0; m < PAIRS; ++m)
      S[c][m] = f2_pack(live[c] && channel(2 * m) < d ? *state_at(2 * m, c) : 0.f,
                        live[c] && channel(2 * m + 1) < d ? *state_at(2 * m + 1, c) : 0.f);
  for (int e = tid; e < WALK_STAGES * STAGE; e += WALK_THREADS) walk_smem[e] = 0.f;      // channels >= d and columns >= dv stay 0
  __syncthreads();

  const int n_stages = (n + WALK_STAGE - 1) / WALK_STAGE, place0 = walk_place(t0, req);
  const bool wide = d % 4 == 0, wide_v = dv % 4 == 0;      // every row then starts on a 16-byte boundary
  const float* planes[4] = {p.q, p.k, p.kb, p.ab};
  auto load = [&](int stage) {
    float* base = walk_smem + (stage % WALK_STAGES) * STAGE;
    const int first = stage * WALK_STAGE, have = min(WALK_STAGE, n - first);
    const float* src_at[ROWS];
    long long step[ROWS];
#pragma unroll
    for (int a = 0; a < ROWS; ++a) {
      step[a] = a == 0 ? p.q_stride : (a == 1 ? p.k_stride : p.b_stride);
      src_at[a] = planes[a] + (size_t)(t0 + first) * step[a] + (size_t)kh * d;
    }
    const float* w_at = CHANNEL ? p.w + ((size_t)(place0 + 2 * stage) * p.n_heads + head) * d : nullptr;
    if (wide) {
      constexpr int PIECES = DMAX / 4, PASS = WALK_THREADS / PIECES;      // rows a pass of the block fills
      const int piece = tid % PIECES, r0 = tid / PIECES;
      if (piece * 4 < d) {
#pragma unroll
        for (int a = 0; a < ROWS; ++a)
#pragma unroll
          for (int tt = 0; tt < WALK_STAGE; tt += PASS) {
            const int t = tt + r0;
            cp_async_16(base + (a * WALK_STAGE + t) * DMAX + piece * 4,
                        t < have ? src_at[a] + t * step[a] + piece * 4 : src_at[a], t < have ? 16 : 0);
          }
        if (CHANNEL && r0 < 2) {
          const bool there = r0 * WALK_TURN < have;
          cp_async_16(base + AT_W + r0 * DMAX + piece * 4,
                      w_at + (there ? (size_t)r0 * p.n_heads * d : 0) + piece * 4, there ? 16 : 0);
        }
      }
    } else {
      for (int r = tid / 32; r < ROWS * WALK_STAGE; r += WALK_THREADS / 32) {
        const int a = r / WALK_STAGE, t = r % WALK_STAGE;
        const float* src = planes[a] + (size_t)(t0 + first + t) * (a == 0 ? p.q_stride : (a == 1 ? p.k_stride : p.b_stride)) +
                           (size_t)kh * d;
        for (int i = tid & 31; i < d; i += 32) base[r * DMAX + i] = t < have ? src[i] : 0.f;
      }
      if (CHANNEL)
        for (int i = tid; i < 2 * d; i += WALK_THREADS) {
          const int g = i / d, c = i - g * d;
          base[AT_W + g * DMAX + c] = g * WALK_TURN < have ? w_at[(size_t)g * p.n_heads * d + c] : 0.f;
        }
    }
    if (wide_v) {
      if (tid < WALK_STAGE * 4) {
        const int t = tid >> 2, piece = tid & 3;
        if (col0 + piece * 4 < dv) {
          const float* src = p.v + (size_t)(t0 + first) * p.n_heads * dv + (size_t)head * dv + col0 + piece * 4;
          cp_async_16(base + AT_V + t * WALK_COLS + piece * 4, t < have ? src + (size_t)t * p.n_heads * dv : src,
                      t < have ? 16 : 0);
        }
      }
    } else {
      const int t = tid >> 4, c = tid & 15;
      if (col0 + c < dv)
        base[AT_V + t * WALK_COLS + c] =
            t < have ? p.v[(size_t)(t0 + first + t) * p.n_heads * dv + (size_t)head * dv + col0 + c] : 0.f;
    }
    constexpr int TP = TAB / 4;
    if (tid >= 64 && tid < 64 + 2 * TP) {
      const int g = (tid - 64) / TP, piece = (tid - 64) % TP;
      const bool there = g * WALK_TURN < have;
      const float* src = p.tables + ((size_t)(place0 + 2 * stage + (there ? g : 0)) * p.n_heads + head) * TAB + piece * 4;
      cp_async_16(base + AT_T + g * TAB + piece * 4, src, there ? 16 : 0);
    }
    cp_async_commit();
  };

#pragma unroll
  for (int s = 0; s < WALK_STAGES - 1; ++s) {
    if (s < n_stages) load(s);
    else cp_async_commit();
  }
  // The token of a turn and the column whose sum this lane ends with.
  const int mine = (part >> 1) & 3, my_c = part & 1;
  const unsigned keep1 = mine < 1 ? 0u : ~0u, keep2 = mine < 2 ? 0u : ~0u, keep3 = mine < 3 ? 0u : ~0u;
  const bool my_norm = norm[my_c], writes = part < 8 && live[my_c];
  const float my_skip = p.skip ? p.skip[head] : 0.f;
  float* o_at = my_norm ? p.nq + (size_t)t0 * p.n_heads + head : p.o_raw + ((size_t)t0 * p.n_heads + head) * dv + col + my_c;
  const size_t o_step = my_norm ? (size_t)p.n_heads : (size_t)p.n_heads * dv;
  const unsigned group = tid & 16;      // the first lane of this thread's sixteen

  auto turn = [&](const float* base, int g, int first) {
    const float* tab = base + AT_T + g * TAB;
    auto piece = [&](int a, int t, int m) {      // pairs m and m + 1 of token t's row
      return *reinterpret_cast<const ulonglong2*>(base + (a * WALK_STAGE + g * WALK_TURN + t) * DMAX + part * 4 +
                                                  (m / 2) * 4 * WALK_LANES);
    };
    float v[2][4], y[2][4];      // y: what the tokens write (x for GENERAL)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 in = *reinterpret_cast<const float2*>(base + AT_V + (g * WALK_TURN + t) * WALK_COLS + c0);
      v[0][t] = in.x;
      v[1][t] = in.y;
    }
    f2 kr[KEEP ? 4 : 1][PAIRS];      // the rows read for the products are the rows written
    auto dots = [&](int a, float (&out)[8]) {      // token t, column c at 2 t + c: eight chains side by side
      f2 acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};        // pairs of zeros
#pragma unroll
      for (int m = 0; m < PAIRS; m += 2) {
        ulonglong2 r[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) r[t] = piece(a, t, m);
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int c = 0; c < 2; ++c) acc[2 * t + c] = f2_fma(r[t].x, S[c][m], acc[2 * t + c]);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
          for (int c = 0; c < 2; ++c) acc[2 * t + c] = f2_fma(r[t].y, S[c][m + 1], acc[2 * t + c]);
          if (KEEP && a == 1) {
            kr[KEEP ? t : 0][m] = r[t].x;
            kr[KEEP ? t : 0][m + 1] = r[t].y;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = f2_sum(acc[i]);
    };
    float qd[8];
    if constexpr (MODE == WALK_LINEAR) {
      dots(0, qd);
      const float4 gain = *reinterpret_cast<const float4*>(tab + WALK_BETA);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        y[c][0] = norm[c] ? gain.x : v[c][0] * gain.x;
        y[c][1] = norm[c] ? gain.y : v[c][1] * gain.y;
        y[c][2] = norm[c] ? gain.z : v[c][2] * gain.z;
        y[c][3] = norm[c] ? gain.w : v[c][3] * gain.w;
      }
    } else {
      float kd[8], all[8];
      dots(1, kd);
      const float sum = walk_sum8(kd, part);
      dots(0, qd);      // under the shuffles
#pragma unroll
      for (int i = 0; i < 8; ++i) all[i] = __shfl_sync(0xffffffffu, sum, group + i);
      if constexpr (MODE == WALK_GENERAL) {
        const float4 a0 = *reinterpret_cast<const float4*>(tab + WALK_GA), b0 = *reinterpret_cast<const float4*>(tab + WALK_GB);
        const float2 a1 = *reinterpret_cast<const float2*>(tab + WALK_GA + 4), b1 = *reinterpret_cast<const float2*>(tab + WALK_GB + 4);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          y[c][0] = all[c];
          y[c][1] = fmaf(a0.x, y[c][0], fmaf(b0.x, v[c][0], all[2 + c]));
          y[c][2] = fmaf(a0.z, y[c][1], fmaf(a0.y, y[c][0], fmaf(b0.z, v[c][1], fmaf(b0.y, v[c][0], all[4 + c]))));
          y[c][3] = fmaf(a1.y, y[c][2], fmaf(a1.x, y[c][1], fmaf(a0.w, y[c][0],
                    fmaf(b1.y, v[c][2], fmaf(b1.x, v[c][1], fmaf(b0.w, v[c][0], all[6 + c]))))));
        }
      } else {
        const float4 P = *reinterpret_cast<const float4*>(tab + WALK_P), be = *reinterpret_cast<const float4*>(tab + WALK_BETA);
        const float4 k0 = *reinterpret_cast<const float4*>(tab + WALK_K);
        const float2 k1 = *reinterpret_cast<const float2*>(tab + WALK_K + 4);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          y[c][0] = be.x * fmaf(-P.x, all[c], v[c][0]);
          y[c][1] = be.y * fmaf(-k0.x, y[c][0], fmaf(-P.y, all[2 + c], v[c][1]));
          y[c][2] = be.z * fmaf(-k0.z, y[c][1], fmaf(-k0.y, y[c][0], fmaf(-P.z, all[4 + c], v[c][2])));
          y[c][3] = be.w * fmaf(-k1.y, y[c][2], fmaf(-k1.x, y[c][1], fmaf(-k0.w, y[c][0], fmaf(-P.w, all[6 + c], v[c][3]))));
        }
      }
    }
    // The state at the turn's end.
    if constexpr (CHANNEL) {
#pragma unroll
      for (int m = 0; m < PAIRS; m += 2) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(base + AT_W + g * DMAX + part * 4 + (m / 2) * 4 * WALK_LANES);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[c][m] = f2_mul(S[c][m], w.x);
          S[c][m + 1] = f2_mul(S[c][m + 1], w.y);
        }
      }
    } else {
      const float whole = tab[WALK_P + 3];
      const f2 w = f2_pack(whole, whole);
#pragma unroll
      for (int m = 0; m < PAIRS; ++m)
#pragma unroll
        for (int c = 0; c < 2; ++c) S[c][m] = f2_mul(S[c][m], w);
    }
    float z[4] = {1.f, 1.f, 1.f, 1.f};
    if constexpr (!CHANNEL) {
      const float4 Z = *reinterpret_cast<const float4*>(tab + WALK_Z);
      z[0] = Z.x; z[1] = Z.y; z[2] = Z.z; z[3] = Z.w;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      // GENERAL writes k v and a x, the others k y.
      f2 ys[2], xs[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float s = MODE == WALK_GENERAL ? v[c][t] : (CHANNEL ? y[c][t] : z[t] * y[c][t]);
        ys[c] = f2_pack(s, s);
        xs[c] = f2_pack(y[c][t], y[c][t]);
      }
#pragma unroll
      for (int m = 0; m < PAIRS; m += 2) {
        ulonglong2 r;
        if constexpr (KEEP) {
          r.x = kr[t][m];
          r.y = kr[t][m + 1];
        } else {
          r = piece(MODE == WALK_LINEAR || MODE == WALK_GATED ? 1 : 2, t, m);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[c][m] = f2_fma(r.x, ys[c], S[c][m]);
          S[c][m + 1] = f2_fma(r.y, ys[c], S[c][m + 1]);
        }
        if constexpr (MODE == WALK_GENERAL) {
          const ulonglong2 a = piece(3, t, m);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            S[c][m] = f2_fma(a.x, xs[c], S[c][m]);
            S[c][m + 1] = f2_fma(a.y, xs[c], S[c][m + 1]);
          }
        }
      }
    }
    // The read-outs.
    float o = walk_sum8(qd, part);
    if (!CHANNEL) o *= tab[WALK_P + mine];
    const float4 Q = *reinterpret_cast<const float4*>(tab + (MODE == WALK_GENERAL ? WALK_GQ : WALK_Q) + 4 * mine);
    o = fmaf(Q.w, walk_keep(my_c ? y[1][3] : y[0][3], keep3), fmaf(Q.z, walk_keep(my_c ? y[1][2] : y[0][2], keep2),
        fmaf(Q.y, walk_keep(my_c ? y[1][1] : y[0][1], keep1), fmaf(Q.x, my_c ? y[1][0] : y[0][0], o))));
    if constexpr (MODE == WALK_GENERAL) {
      const float4 R = *reinterpret_cast<const float4*>(tab + WALK_GR + 4 * mine);
      o = fmaf(R.w, walk_keep(my_c ? v[1][3] : v[0][3], keep3), fmaf(R.z, walk_keep(my_c ? v[1][2] : v[0][2], keep2),
          fmaf(R.y, walk_keep(my_c ? v[1][1] : v[0][1], keep1), fmaf(R.x, my_c ? v[1][0] : v[0][0], o))));
    }
    if constexpr (MODE == WALK_LINEAR) {
      if (p.skip) o = fmaf(my_skip, base[AT_V + (g * WALK_TURN + mine) * WALK_COLS + c0 + my_c], o);
    }
    if (writes && first + mine < n) o_at[(size_t)(first + mine) * o_step] = o;
  };

  for (int it = 0; it < n_stages; ++it) {
    cp_async_wait<WALK_STAGES - 2>();
    __syncthreads();      // the stage is there for everyone, and everyone is done with the one that is filled next
    if (it + WALK_STAGES - 1 < n_stages) load(it + WALK_STAGES - 1);
    else cp_async_commit();
    const float* base = walk_smem + (it % WALK_STAGES) * STAGE;
    const int first = it * WALK_STAGE;
    if (first + WALK_TURN < n) {
      turn(base, 0, first);
      turn(base, 1, first + WALK_TURN);
    } else {
      turn(base, 0, first);
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if (live[c]) {
#pragma unroll
      for (int m = 0; m < PAIRS; ++m) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(S[c][m]));
        if (channel(2 * m) < d) *state_at(2 * m, c) = lo;
        if (channel(2 * m + 1) < d) *state_at(2 * m + 1, c) = hi;
      }
    }
}

// A turn's coefficients from the products of its rows, summed over the warp: lane l < 16 has sum l (q_i . k_j, j <= i, at
// i (i + 1) / 2 + j; k_i . k_j, j < i, at 10 + i (i - 1) / 2 + j). g: the tokens' decays, be: their write strengths or gains.
// With a decay per key channel the sums hold the decays already (and g is ones).
template <int MODE>
__device__ __forceinline__ void walk_write_table(float* __restrict__ to, float sum, const float (&g)[4], const float (&be)[4],
                                                 int lane) {
  // Lane l < 16 holds sum l: its factor is the decays after j up to and with i.
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float between = 1.f;
#pragma unroll
    for (int j = i; j >= 0; --j) {
      if (lane == i * (i + 1) / 2 + j) to[WALK_Q + 4 * i + j] = sum * between;
      if (MODE != WALK_LINEAR && j < i && lane == 10 + i * (i - 1) / 2 + j) to[WALK_K + i * (i - 1) / 2 + j] = sum * between;
      between *= g[j];
    }
  }
  const float p1 = g[0] * g[1], p2 = p1 * g[2], z1 = g[3] * g[2], z0 = z1 * g[1];
  if (lane == 16) *reinterpret_cast<float4*>(to + WALK_P) = make_float4(g[0], p1, p2, p2 * g[3]);
  if (lane == 17) *reinterpret_cast<float4*>(to + WALK_Z) = make_float4(z0, z1, g[3], 1.f);
  if (lane == 18) *reinterpret_cast<float4*>(to + WALK_BETA) = make_float4(be[0], be[1], be[2], be[3]);
  if (lane >= 19 && lane < 25) {      // above the diagonal
    const int e = lane - 19, at = e < 3 ? 1 + e : (e < 5 ? 3 + e : 11);      // (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
    to[WALK_Q + at] = 0.f;
  }
}

// The coefficients of WALK_LINEAR (a decay per token and head): a warp per (turn, head). decay [tokens, heads]
// or null (then head_decay [heads], or 1); beta [tokens, heads] or null (1): gains on the values.
template <int CPL>
__global__ void __launch_bounds__(128)
walk_tables_kernel(const float* __restrict__ q, const float* __restrict__ k, long long stride, const float* __restrict__ decay,
                   const float* __restrict__ head_decay, const float* __restrict__ beta, const int* __restrict__ q_start,
                   const int* __restrict__ n_new, float* __restrict__ tables, int n_requests, int n_heads, int n_groups, int d,
                   int from) {
  const int place = blockIdx.x, head = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (head >= n_heads) return;
  const int req = walk_request(q_start, n_requests, place), t_req = q_start[req];
  const int first = (place - walk_place(t_req, req)) * WALK_TURN, have = min(WALK_TURN, n_new[req] - first);
  if (first < 0 || have <= 0 || n_new[req] < from) return;
  const size_t t0 = (size_t)(t_req + first);
  const float* qr = q + t0 * stride + (size_t)(head / (n_heads / n_groups)) * d;
  const float* kr = k + t0 * stride + (size_t)(head / (n_heads / n_groups)) * d;
  float sums[16];      // q_i . k_j (j <= i) at i (i + 1) / 2 + j
#pragma unroll
  for (int e = 0; e < 16; ++e) sums[e] = 0.f;
  float qv[4][CPL], kv[4][CPL];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    walk_load<CPL>(qr + t * stride, lane, d, t < have, d % 4 == 0, qv[t]);
    walk_load<CPL>(kr + t * stride, lane, d, t < have, d % 4 == 0, kv[t]);
  }
  float g[4], be[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    g[t] = t >= have ? 1.f : (decay ? decay[(t0 + t) * n_heads + head] : (head_decay ? head_decay[head] : 1.f));
    be[t] = t >= have ? 0.f : (beta ? beta[(t0 + t) * n_heads + head] : 1.f);
  }
#pragma unroll
  for (int m = 0; m < CPL; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) sums[i * (i + 1) / 2 + j] = fmaf(qv[i][m], kv[j][m], sums[i * (i + 1) / 2 + j]);
  walk_write_table<WALK_LINEAR>(tables + ((size_t)place * n_heads + head) * 36, walk_sum_all<16>(sums, lane), g, be, lane);
}

static int launch_walk_tables(const float* q, const float* k, long long stride, const float* decay, const float* head_decay,
                              const float* beta, const int* q_start, const int* n_new, float* tables, int n_tokens,
                              int n_requests, int n_heads, int n_groups, int d, int from, cudaStream_t stream) {
  const dim3 grid((unsigned)walk_places(n_tokens, n_requests), (n_heads + 3) / 4);
  if (d <= 128)
    walk_tables_kernel<4><<<grid, 128, 0, stream>>>(q, k, stride, decay, head_decay, beta, q_start, n_new, tables,
                                                    n_requests, n_heads, n_groups, d, from);
  else
    walk_tables_kernel<8><<<grid, 128, 0, stream>>>(q, k, stride, decay, head_decay, beta, q_start, n_new, tables,
                                                    n_requests, n_heads, n_groups, d, from);
  return llmrs_launch_status("state walk (tables)");
}

template <int MODE, int DMAX, bool SOME>
static int launch_state_walk_of(const WalkArgs& a, int n_requests, int cols, cudaStream_t stream) {
  constexpr size_t smem = (size_t)WALK_STAGES * walk_stage_floats(MODE, DMAX) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(state_walk_kernel<MODE, DMAX, SOME>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return llmrs_fail("state walk: shared memory %zu: %s", smem, cudaGetErrorString(e));
  }
  const int col_blocks = (cols + WALK_COLS - 1) / WALK_COLS;
  const long long blocks = (long long)n_requests * a.n_heads * col_blocks;
  LLMRS_REQUIRE(blocks <= 0x7fffffffLL, "state walk: too many requests, heads or columns");
  state_walk_kernel<MODE, DMAX, SOME><<<(unsigned)blocks, WALK_THREADS, smem, stream>>>(a, col_blocks);
  return llmrs_launch_status("state walk");
}

// cols: value columns, the normaliser's among them.
template <int MODE>
static int launch_state_walk(const WalkArgs& a, int n_requests, int cols, cudaStream_t stream) {
#define LLMRS_WALK(D) \
  return a.from > 1 ? launch_state_walk_of<MODE, D, true>(a, n_requests, cols, stream) : launch_state_walk_of<MODE, D, false>(a, n_requests, cols, stream)
  if (a.d <= 64) LLMRS_WALK(64);
  if (a.d <= 128) LLMRS_WALK(128);
  LLMRS_WALK(256);
#undef LLMRS_WALK
}
