// Gated delta rule: a recurrent mixer with a matrix state S [key channel, value channel] per head,
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (the read-out sees the token's own write)
//
// beta in (0, 1) is one number per head and token; the decay g in (0, 1) is one number per head and token, or one per
// head, token and KEY CHANNEL (g then multiplies the rows of S, S[i, :] <- g[i] S[i, :]). q and k (G heads of d channels; value head h reads
// q/k head h / (H / G)) and v (H heads of dv channels) each pass a short causal convolution over time per channel
// (K taps, the last one the current token's, zeros before a sequence's start) and SiLU; q and k are then made unit
// vectors per head (x / sqrt(sum x^2 + key_eps)), q is also multiplied by q_scale. g = exp(-exp(A_log_h) *
// softplus(a + dt_bias_h)) and beta = sigmoid(b) come from two float32 projections a, b. After the recurrence each head's
// o is divided by its root mean square over dv, multiplied by a weight of size dv (shared by the heads) and by
// SiLU(gate) or sigmoid(gate). With a decay per key channel the raw decay a [tokens, H d] already holds a number per
// channel, dt_bias has one too (A_log stays one per head), and b comes in the activation type. Everything but the
// projections' inputs is float32.
//
// Per-request state: S (float32 [slots, H, d, dv]) and the last K - 1 rows that entered the convolutions
// (float32 [slots, K - 1, C], C = 2 G d + H dv: the q, k and v channels side by side, oldest row first).
//
//   prepare      a block per token: convolutions + SiLU, unit q and k, g and beta, as float32 rows
//   conv state   a block per request, after prepare: the request's last K - 1 convolution inputs
//   (requests that are walked: rows by one kernel in place of `prepare`, then, heads of up to 128 channels, the chunks' rows and
//   the walk of state_chunks.cuh; others the coefficients of turns of four tokens with the rows and the walk of state_walk.cuh)
//   recurrence   of the others, token by token: a block per (request, head, slice of 16 value
//                columns) walks the request's tokens; four
//                neighbouring lanes share a column, each with a quarter of the key channels in registers (lane p of the
//                four holds channels 4 (p + 4 j) .. 4 (p + 4 j) + 3, so that the four read neighbouring 16-byte pieces
//                of a row in shared memory, not pieces a bank's stride apart); k^T S and q^T S are summed over the four
//                by two shuffles. Rows come in chunks through two shared-memory buffers.
//   output       norm, weight, gate (head_out.cuh; heads that it does not take: a warp per token and head)
//
// Long portions may take the recurrence in CHUNKS of 32 tokens instead (the same numbers up to float32 rounding, all of it
// float32 FMA). Within a chunk that starts from the state S_0, with L_t the sum of log g up to and including token t:
//
//   u_t = beta_t (v_t - e^{L_t} S_0^T k_t - sum_{s<t} A[t,s] u_s),     A[t,s] = e^{L_t - L_s} (k_t . k_s)
//   =>  U = T (V - diag(e^L) K S_0),   T = (I + diag(beta) A)^{-1} diag(beta)      (32 x 32, lower triangular)
//   o_t = e^{L_t} S_0^T q_t + sum_{s<=t} P[t,s] u_s,                    P[t,s] = e^{L_t - L_s} (q_t . k_s)
//   S_32 = e^{L_32} S_0 + K^T diag(e^{L_32 - L_s}) U
//
// T, P and the decays depend on no state: `chunk tables` makes them for every chunk and head at once (a block each).
// `chunked recurrence` then walks a request's chunks with a block per (request, head, 16 value columns): five small
// products per chunk over rows that arrive through two shared-memory buffers, 32 tokens per sequential step instead of
// one. A chunk's missing tokens (a portion's end) count as k = q = v = 0, beta = 0, g = 1 and change nothing.
// The chunked form is OFF by default (llmrs_gated_delta_chunked): its products read every operand from shared memory
// and are bound by that (2,048 tokens of 16 heads of 128 x 128: some 500 us, the walk in turns 265, in chunks on the tensor cores 117).
#include <limits.h>

#include "common.cuh"
#include "head_out.cuh"
#include "mma_util.cuh"
#include "short_conv.cuh"
#include "state_chunks.cuh"

// CHANNEL: a decay per key channel; ba is then unused, b (activation type) and araw (float32 [tokens, H d]) take its place
// and pg is [tokens, H d].
template <typename TA, bool CHANNEL>
__global__ void gdr_prepare_kernel(const TA* __restrict__ x, long long stride, const float* __restrict__ taps,
                                   const float* __restrict__ ba, const TA* __restrict__ b, long long b_stride,
                                   const float* __restrict__ araw, const float* __restrict__ a_log,
                                   const float* __restrict__ dt_bias, const float* __restrict__ conv_state,
                                   const int* __restrict__ token_req, const int* __restrict__ q_start,
                                   const int* __restrict__ n_new, const int* __restrict__ slot_ids,
                                   float* __restrict__ pq, float* __restrict__ pk, float* __restrict__ pv,
                                   float* __restrict__ pbeta, float* __restrict__ pg, float* __restrict__ plg, int G, int H,
                                   int d, int dv, int K, float key_eps, float q_scale, int below) {
  extern __shared__ float row[];      // [C] after convolution and SiLU
  const int t = blockIdx.x, req = token_req[t], off = t - q_start[req];
  if (below < INT_MAX && n_new[req] >= below) return;      // walked in turns
  const int wq = G * d, wv = H * dv, C = 2 * wq + wv;
  const float* tail = conv_state + (size_t)slot_ids[req] * (K - 1) * C;
  for (int c = threadIdx.x; c < C; c += blockDim.x)
    row[c] = rec_silu(short_conv_at(x, stride, t, off, c, taps + (size_t)c * K, K, tail, C, 0.f));
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int hh = warp; hh < 2 * G; hh += nwarps) {      // q heads, then k heads
    const float* src = row + (size_t)hh * d;
    float ss = 0.f;
    for (int i = lane; i < d; i += 32) ss = fmaf(src[i], src[i], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) + key_eps) * (hh < G ? q_scale : 1.0f);
    float* dst = hh < G ? pq + (size_t)t * wq + (size_t)hh * d : pk + (size_t)t * wq + (size_t)(hh - G) * d;
    for (int i = lane; i < d; i += 32) dst[i] = src[i] * inv;
  }
  for (int c = threadIdx.x; c < wv; c += blockDim.x) pv[(size_t)t * wv + c] = row[2 * wq + c];
  if constexpr (CHANNEL) {
    for (int h = threadIdx.x; h < H; h += blockDim.x)
      pbeta[(size_t)t * H + h] = rec_sigmoid(to_float(b[(size_t)t * b_stride + h]));
    for (int c = threadIdx.x; c < H * d; c += blockDim.x)
      pg[(size_t)t * H * d + c] = expf(-expf(a_log[c / d]) * rec_softplus(araw[(size_t)t * H * d + c] + dt_bias[c]));
  } else {
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
      pbeta[(size_t)t * H + h] = rec_sigmoid(ba[(size_t)t * 2 * H + h]);
      const float lg = -expf(a_log[h]) * rec_softplus(ba[(size_t)t * 2 * H + H + h] + dt_bias[h]);      // log g
      plg[(size_t)t * H + h] = lg;
      pg[(size_t)t * H + h] = expf(lg);
    }
  }
}

constexpr int GD_COLS = 16;      // value columns of a block
#ifndef LLMRS_GD_LANES
#define LLMRS_GD_LANES 8
#endif
// (The kernel that walks token by token.) With a decay per key channel a lane reads three rows a
// token, not two: sixteen lanes a column shorten that where a step's blocks do not fill the device twice (walking 2,048 tokens
// of 16 heads of 128 x 128: 813 against 896 us for the whole op), eight are ahead where they do.
constexpr int GD_WIDE_MAX_BLOCKS = 296;

// LANES: neighbouring lanes that share a column (4, 8 or 16; at most DMAX / 4, so that a lane holds whole pieces of
// four channels). CHANNEL: pg holds a decay per key channel, [tokens, H d], which travels like q and k.
// SOME: only requests of fewer than `below` tokens, the others are walked in turns (a template: the test alone cost decode steps
// of 200 requests 2 %).
template <int DMAX, int LANES, bool CHANNEL, bool SOME>
__global__ void __launch_bounds__(GD_COLS * LANES)
gdr_recurrence_kernel(const float* __restrict__ pq, const float* __restrict__ pk, const float* __restrict__ pv,
                      const float* __restrict__ pbeta, const float* __restrict__ pg, float* __restrict__ state,
                      const int* __restrict__ q_start, const int* __restrict__ n_new,
                      const int* __restrict__ slot_ids, float* __restrict__ o_raw, int G, int H, int d, int dv, int below) {
  constexpr int CHUNK = CHANNEL ? (DMAX >= 256 ? 4 : (DMAX >= 128 ? 8 : 16)) : (DMAX >= 256 ? 8 : 16);
  constexpr int PLANES = CHANNEL ? 3 : 2;
  constexpr int GD_LANES = LANES, GD_THREADS = GD_COLS * LANES;
  constexpr int IPL = DMAX / GD_LANES;             // key channels per lane
  __shared__ __align__(16) float s_qk[2][PLANES][CHUNK][DMAX];      // q, k (and g) of a chunk's tokens; channels >= d stay 0
  __shared__ float s_v[2][CHUNK][GD_COLS], s_bg[2][2][CHUNK];
  // The lanes' shares of a chunk's read-outs: summed over a column's lanes after the chunk's walk, by all threads at
  // once, instead of by a chain of shuffles in every token's turn (the walk then waits for one such chain a token,
  // the one it cannot do without: k^T S).
  __shared__ float s_o[CHUNK][GD_COLS][LANES + 1];
  const int req = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * GD_COLS;
  const int kh = head / (H / G);
  const int tid = threadIdx.x;
  const int col = col0 + tid / GD_LANES, part = tid % GD_LANES;
  // Register i of a lane holds key channel ch(i): pieces of four channels dealt out to the four lanes in turn.
  auto ch = [&](int i) { return ((i >> 2) * GD_LANES + part) * 4 + (i & 3); };
  const bool live = col < dv;
  const int t0 = q_start[req], n = n_new[req];
  if (SOME && n >= below) return;
  const int wq = G * d, wv = H * dv;
  float* S_g = state + ((size_t)slot_ids[req] * H + head) * d * dv;
  float S[IPL];
#pragma unroll
  for (int i = 0; i < IPL; ++i) S[i] = (live && ch(i) < d) ? S_g[(size_t)ch(i) * dv + col] : 0.f;
  for (int e = tid; e < 2 * PLANES * CHUNK * DMAX; e += GD_THREADS) (&s_qk[0][0][0][0])[e] = 0.f;
  for (int e = tid; e < 2 * CHUNK * GD_COLS; e += GD_THREADS) (&s_v[0][0][0])[e] = 0.f;
  __syncthreads();
  const bool wide = d % 4 == 0;      // every row then starts on a 16-byte boundary
  const int ncols = min(GD_COLS, dv - col0);
  auto load_chunk = [&](int buf, int c0) {
    const int cn = min(CHUNK, n - c0);
    auto row_of = [&](int a, int tt) {
      const size_t t = (size_t)(t0 + c0 + tt);
      if (CHANNEL && a == 2) return pg + t * H * d + (size_t)head * d;
      return (a == 0 ? pq : pk) + t * wq + (size_t)kh * d;
    };
    if (wide) {
      const int per_row = d / 4;
      for (int e = tid; e < PLANES * cn * per_row; e += GD_THREADS) {
        const int a = e / (cn * per_row), rem = e % (cn * per_row), tt = rem / per_row, piece = rem % per_row;
        cp_async_16(&s_qk[buf][a][tt][piece * 4], row_of(a, tt) + piece * 4, 16);
      }
    } else {
      for (int e = tid; e < PLANES * cn * d; e += GD_THREADS) {
        const int a = e / (cn * d), rem = e % (cn * d), tt = rem / d, i = rem % d;
        s_qk[buf][a][tt][i] = row_of(a, tt)[i];
      }
    }
    // (Values and gates by asynchronous copies too: a plain load would hold the warp for a memory round trip at the top
    // of every chunk, before it starts on the tokens it already has.)
    for (int e = tid; e < cn * ncols; e += GD_THREADS) {
      const int tt = e / ncols, c = e % ncols;
      cp_async_4(&s_v[buf][tt][c], pv + (size_t)(t0 + c0 + tt) * wv + (size_t)head * dv + col0 + c);
    }
    for (int e = tid; e < (CHANNEL ? 1 : 2) * cn; e += GD_THREADS) {
      const int a = e / cn, tt = e % cn;
      cp_async_4(&s_bg[buf][a][tt], (a == 0 ? pbeta : pg) + (size_t)(t0 + c0 + tt) * H + head);
    }
    cp_async_commit();
  };

  if (n > 0) load_chunk(0, 0);
  for (int c0 = 0, it = 0; c0 < n; c0 += CHUNK, ++it) {
    const int cn = min(CHUNK, n - c0), buf = it & 1;
    if (c0 + CHUNK < n) {
      load_chunk(buf ^ 1, c0 + CHUNK);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll 4
    for (int tt = 0; tt < cn; ++tt) {
      const float vj = s_v[buf][tt][tid / GD_LANES], beta = s_bg[buf][0][tt], g = CHANNEL ? 1.0f : s_bg[buf][1][tt];
      float ks[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < IPL; i += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&s_qk[buf][1][tt][ch(i)]);
        if constexpr (CHANNEL) {
          const float4 g4 = *reinterpret_cast<const float4*>(&s_qk[buf][2][tt][ch(i)]);
          S[i] *= g4.x; S[i + 1] *= g4.y; S[i + 2] *= g4.z; S[i + 3] *= g4.w;
        } else {
          S[i] *= g; S[i + 1] *= g; S[i + 2] *= g; S[i + 3] *= g;
        }
        ks[0] = fmaf(k4.x, S[i], ks[0]);
        ks[1] = fmaf(k4.y, S[i + 1], ks[1]);
        ks[2] = fmaf(k4.z, S[i + 2], ks[2]);
        ks[3] = fmaf(k4.w, S[i + 3], ks[3]);
      }
      float kS = (ks[0] + ks[1]) + (ks[2] + ks[3]);
#pragma unroll
      for (int off = 1; off < LANES; off <<= 1) kS += __shfl_xor_sync(0xffffffffu, kS, off);
      const float u = beta * (vj - kS);
      float os[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < IPL; i += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&s_qk[buf][1][tt][ch(i)]);
        const float4 q4 = *reinterpret_cast<const float4*>(&s_qk[buf][0][tt][ch(i)]);
        S[i] = fmaf(k4.x, u, S[i]);
        S[i + 1] = fmaf(k4.y, u, S[i + 1]);
        S[i + 2] = fmaf(k4.z, u, S[i + 2]);
        S[i + 3] = fmaf(k4.w, u, S[i + 3]);
        os[0] = fmaf(S[i], q4.x, os[0]);
        os[1] = fmaf(S[i + 1], q4.y, os[1]);
        os[2] = fmaf(S[i + 2], q4.z, os[2]);
        os[3] = fmaf(S[i + 3], q4.w, os[3]);
      }
      s_o[tt][tid / GD_LANES][part] = (os[0] + os[1]) + (os[2] + os[3]);
    }
    __syncthreads();
    for (int e = tid; e < cn * GD_COLS; e += GD_THREADS) {
      const int tt = e / GD_COLS, c = e % GD_COLS;
      float o = 0.f;
#pragma unroll
      for (int p = 0; p < LANES; ++p) o += s_o[tt][c][p];
      if (col0 + c < dv) o_raw[(size_t)(t0 + c0 + tt) * wv + (size_t)head * dv + col0 + c] = o;
    }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < IPL; ++i)
      if (ch(i) < d) S_g[(size_t)ch(i) * dv + col] = S[i];
  }
}


// ---- the walk in turns of four tokens (state_walk.cuh) ---------------------------------------------------------------
// What it reads, made from the projections' rows in one kernel: a warp per (turn, key head) or (turn, 32 CPL value channels).
// A key head's warp convolves its q and k for the turn's four tokens (the seven rows they need and four taps a channel in
// registers), makes them unit vectors and, for every value head that shares them, the coefficients between the tokens. With a
// decay per key channel it leaves the rows with their decays instead (qf, kf from the turn's start up to and with the token,
// kb from the token to the turn's end) and the whole turn's decay. Products of decays, no quotients: nothing overflows.
// Six blocks an SM take 51 us, four 58. 2,048 tokens of 16 heads over 8 of 128 x 128: 51 us, where preparing the rows (a block a token, the
// convolution a channel at a time) and their coefficients by two kernels took 68 + 13.
template <int CPL, typename TA>
__device__ __forceinline__ void gdr_convolve(const TA* __restrict__ x, long long stride, size_t t_req, int first, int have,
                                             const float* __restrict__ taps, int K, bool taps4, const float* __restrict__ tail,
                                             int C, int lane, int width, bool vec, float (&out)[4][CPL]) {
  constexpr int V = CPL < 4 ? CPL : 4;
  float in[7][CPL], w[4][CPL];      // the rows of tokens first - 3 .. first + 3; the taps of lags 0 .. 3
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const int o = first - 3 + i;
    if (o >= 0) walk_load<CPL>(x + (t_req + o) * stride, lane, width, o < first + have, vec, in[i]);
    else walk_load<CPL>(tail + (long long)(K - 1 + o) * C, lane, width, K - 1 + o >= 0, vec, in[i]);
  }
#pragma unroll
  for (int m = 0; m < CPL; ++m) {
    const int c = V * lane + 32 * (m / V * V) + m % V;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);      // lags 3, 2, 1, 0
    if (c < width) {
      const float* at = taps + (size_t)c * K;
      if (taps4) {
        f = *reinterpret_cast<const float4*>(at);
      } else {
        f.w = at[K - 1];
        if (K > 1) f.z = at[K - 2];
        if (K > 2) f.y = at[K - 3];
        if (K > 3) f.x = at[K - 4];
      }
    }
    w[0][m] = f.w; w[1][m] = f.z; w[2][m] = f.y; w[3][m] = f.x;
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float acc[CPL];
#pragma unroll
    for (int m = 0; m < CPL; ++m) acc[m] = 0.f;
#pragma unroll
    for (int lag = 0; lag < 4; ++lag)
      if (lag < K)
#pragma unroll
        for (int m = 0; m < CPL; ++m) acc[m] = fmaf(w[lag][m], in[3 + t - lag][m], acc[m]);
    for (int lag = 4; lag < K; ++lag) {      // (longer filters: the row and the tap from memory)
      const int o = first + t - lag;
      float row[CPL];
      if (o >= 0) walk_load<CPL>(x + (t_req + o) * stride, lane, width, t < have, vec, row);
      else walk_load<CPL>(tail + (long long)(K - 1 + o) * C, lane, width, t < have, vec, row);
#pragma unroll
      for (int m = 0; m < CPL; ++m) {
        const int c = V * lane + 32 * (m / V * V) + m % V;
        if (c < width) acc[m] = fmaf(taps[(size_t)c * K + K - 1 - lag], row[m], acc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < CPL; ++m) out[t][m] = t < have ? rec_silu(acc[m]) : 0.f;
  }
}

template <typename TA, int CPL, bool CHANNEL, bool CHUNKS>
__global__ void __launch_bounds__(128, CPL == 4 ? 6 : 1)
gdr_turns_kernel(const TA* __restrict__ x, long long stride, const float* __restrict__ taps, const float* __restrict__ ba,
                 const TA* __restrict__ b, long long b_stride, const float* __restrict__ araw, const float* __restrict__ a_log,
                 const float* __restrict__ dt_bias, const float* __restrict__ conv_state, const int* __restrict__ q_start,
                 const int* __restrict__ n_new, const int* __restrict__ slot_ids, float* __restrict__ pq,
                 float* __restrict__ pk, float* __restrict__ kb, float* __restrict__ pv, float* __restrict__ w,
                 float* __restrict__ tables, float* __restrict__ pbeta, float* __restrict__ pg, int n_requests, int G, int H, int d, int dv, int K, float key_eps, float q_scale,
                 bool vec, bool taps4, int from) {
  const int place = blockIdx.x, unit = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int wq = G * d, wv = H * dv, C = 2 * wq + wv;
  if (unit >= G + (wv + 32 * CPL - 1) / (32 * CPL)) return;
  const int req = walk_request(q_start, n_requests, place), t_req = q_start[req];
  const int first = (place - walk_place(t_req, req)) * WALK_TURN, have = min(WALK_TURN, n_new[req] - first);
  if (first < 0 || have <= 0 || n_new[req] < from) return;
  const size_t t0 = (size_t)(t_req + first);
  const float* tail = conv_state + (size_t)slot_ids[req] * (K - 1) * C;
  auto convolve = [&](int c0, int width, float (&out)[4][CPL]) {
    gdr_convolve<CPL>(x + c0, stride, (size_t)t_req, first, have, taps + (size_t)c0 * K, K, taps4, tail + c0, C, lane, width, vec, out);
  };
  if (unit >= G) {
    const int c0 = (unit - G) * 32 * CPL, width = min(32 * CPL, wv - c0);
    float v[4][CPL];
    convolve(2 * wq + c0, width, v);
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (t < have) walk_store<CPL>(pv + (t0 + t) * wv + c0, lane, width, vec, v[t]);
    return;
  }
  float q[4][CPL], k[4][CPL];
  convolve(unit * d, d, q);
  convolve(wq + unit * d, d, k);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
      sq = fmaf(q[t][m], q[t][m], sq);
      sk = fmaf(k[t][m], k[t][m], sk);
    }
    const float iq = 1.0f / sqrtf(warp_sum(sq) + key_eps) * q_scale, ik = 1.0f / sqrtf(warp_sum(sk) + key_eps);
#pragma unroll
    for (int m = 0; m < CPL; ++m) {      // (a token that is not there stays zero also where key_eps is)
      q[t][m] = t < have ? q[t][m] * iq : 0.f;
      k[t][m] = t < have ? k[t][m] * ik : 0.f;
    }
    if ((CHUNKS || !CHANNEL) && t < have) {
      walk_store<CPL>(pq + (t0 + t) * wq + (size_t)unit * d, lane, d, vec, q[t]);
      walk_store<CPL>(pk + (t0 + t) * wq + (size_t)unit * d, lane, d, vec, k[t]);
    }
  }
  const int shared = H / G;
  if constexpr (CHUNKS) {      // the rows as they are, each token's write strengths and, one a head, decays
    for (int e = lane; e < have * shared; e += 32) {
      const int h = unit * shared + e % shared;
      const size_t at = t0 + e / shared;
      if (CHANNEL) {
        pbeta[at * H + h] = rec_sigmoid(to_float(b[at * b_stride + h]));
      } else {
        pbeta[at * H + h] = rec_sigmoid(ba[at * 2 * H + h]);
        pg[at * H + h] = expf(-expf(a_log[h]) * rec_softplus(ba[at * 2 * H + H + h] + dt_bias[h]));
      }
    }
  } else if constexpr (!CHANNEL) {
    // q_i . k_j (j <= i) at i (i + 1) / 2 + j, k_i . k_j (j < i) at 10 + i (i - 1) / 2 + j.
    float sums[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) sums[e] = 0.f;
#pragma unroll
    for (int m = 0; m < CPL; ++m)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          sums[i * (i + 1) / 2 + j] = fmaf(q[i][m], k[j][m], sums[i * (i + 1) / 2 + j]);
          if (j < i) sums[10 + i * (i - 1) / 2 + j] = fmaf(k[i][m], k[j][m], sums[10 + i * (i - 1) / 2 + j]);
        }
    const float sum = walk_sum_all<16>(sums, lane);
    for (int h = unit * shared; h < (unit + 1) * shared; ++h) {
      float be = 0.f, decay = 1.f;      // of token lane & 3
      if ((lane & 3) < have) {
        const float* at = ba + (t0 + (lane & 3)) * 2 * H + h;
        be = rec_sigmoid(at[0]);
        decay = expf(-expf(a_log[h]) * rec_softplus(at[H] + dt_bias[h]));
      }
      float g[4], bt[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        g[t] = __shfl_sync(0xffffffffu, decay, t);
        bt[t] = __shfl_sync(0xffffffffu, be, t);
      }
      walk_write_table<WALK_GATED>(tables + ((size_t)place * H + h) * 36, sum, g, bt, lane);
    }
  } else {
    for (int h = unit * shared; h < (unit + 1) * shared; ++h) {
      const float rate = -expf(a_log[h]);
      float g[4][CPL], bias[CPL], sums[16];
      walk_load<CPL>(dt_bias + (size_t)h * d, lane, d, true, false, bias);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        walk_load<CPL>(araw + (t0 + t) * H * d + (size_t)h * d, lane, d, t < have, vec, g[t]);
#pragma unroll
        for (int m = 0; m < CPL; ++m) g[t][m] = t < have ? expf(rate * rec_softplus(g[t][m] + bias[m])) : 1.f;
      }
      // The same products with the decays after j up to and with i between them.
#pragma unroll
      for (int e = 0; e < 16; ++e) sums[e] = 0.f;
#pragma unroll
      for (int m = 0; m < CPL; ++m)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float kj = k[j][m];
          sums[j * (j + 1) / 2 + j] = fmaf(q[j][m], kj, sums[j * (j + 1) / 2 + j]);
#pragma unroll
          for (int i = j + 1; i < 4; ++i) {
            kj *= g[i][m];
            sums[i * (i + 1) / 2 + j] = fmaf(q[i][m], kj, sums[i * (i + 1) / 2 + j]);
            sums[10 + i * (i - 1) / 2 + j] = fmaf(k[i][m], kj, sums[10 + i * (i - 1) / 2 + j]);
          }
        }
      float up[CPL], down[CPL], row[CPL];
#pragma unroll
      for (int m = 0; m < CPL; ++m) up[m] = down[m] = 1.f;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int e = 3 - t;
#pragma unroll
        for (int m = 0; m < CPL; ++m) up[m] *= g[t][m];
        if (t < have) {
          const size_t at = ((t0 + t) * H + h) * d;
#pragma unroll
          for (int m = 0; m < CPL; ++m) row[m] = q[t][m] * up[m];
          walk_store<CPL>(pq + at, lane, d, vec, row);
#pragma unroll
          for (int m = 0; m < CPL; ++m) row[m] = k[t][m] * up[m];
          walk_store<CPL>(pk + at, lane, d, vec, row);
        }
        if (e < have) {
#pragma unroll
          for (int m = 0; m < CPL; ++m) row[m] = k[e][m] * down[m];
          walk_store<CPL>(kb + ((t0 + e) * H + h) * d, lane, d, vec, row);
        }
#pragma unroll
        for (int m = 0; m < CPL; ++m) down[m] *= g[e][m];
      }
      walk_store<CPL>(w + ((size_t)place * H + h) * d, lane, d, vec, up);
      const float sum = walk_sum_all<16>(sums, lane);
      const float ones[4] = {1.f, 1.f, 1.f, 1.f};
      float bt[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) bt[t] = t < have ? rec_sigmoid(to_float(b[(t0 + t) * b_stride + h])) : 0.f;
      walk_write_table<WALK_CHANNEL>(tables + ((size_t)place * H + h) * 36, sum, ones, bt, lane);
    }
  }
}

// ---- the walk in chunks of sixteen tokens (state_chunks.cuh) with a decay per key channel ---------------------------------
// A block per (place, head). The coefficients between the tokens are products over the channels with the decays between them: a warp
// walks a token j through the tokens after it, the decays multiplied on as they go (no quotients: nothing overflows), and then token
// 15 - j, so that every warp has seventeen steps. Then sixteen channels and sixteen columns a warp at a time.
constexpr int GCR_THREADS = 256;
__host__ __device__ constexpr int gcr_smem(int dmax) { return 4 * (ck_tile(CK_SYSTEM, dmax) + 3 * CK * (dmax + 4)); }
struct GcrArgs {
  const float *pq, *pk, *pv, *pbeta, *araw, *a_log, *dt_bias;
  const int *q_start, *n_new;
  float *tiles, *u, *g_out;
  int n_requests, G, H, d, dv, from;
};
struct GcrShared {
  alignas(16) __nv_bfloat16 Q[CK_MATRIX], T[CK_MATRIX];
  float sums[2][CK][CK + 1], strength[CK];
};
// True where CAREFUL would make something else of it.
template <int DMAX, bool CAREFUL>
__device__ __forceinline__ bool gdr_channel_rows(const GcrArgs& p, float* tile, GcrShared& sh) {
  constexpr int GS = CK + 1, RS = DMAX + 4, ROW = DMAX + 8, PER = DMAX / 32;
  constexpr int EACH = (CK * (DMAX / 4) + GCR_THREADS - 1) / GCR_THREADS;
  const float *pq = p.pq, *pk = p.pk, *pv = p.pv, *pbeta = p.pbeta, *araw = p.araw, *a_log = p.a_log, *dt_bias = p.dt_bias;
  const int *q_start = p.q_start, *n_new = p.n_new;
  const int n_requests = p.n_requests, G = p.G, H = p.H, d = p.d, dv = p.dv, from = p.from;
  auto q = reinterpret_cast<float (*)[RS]>(tile + ck_tile(CK_SYSTEM, DMAX));
  auto k = q + CK, g = k + CK;
  auto& Q = sh.Q;
  auto& T = sh.T;
  auto& sums = sh.sums;
  auto& strength = sh.strength;
  CkLook look;
  const int place = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int t_req, n_req;
  const int place0 = ck_request(q_start, n_new, n_requests, from, place, t_req, n_req);
  const int first = (place - place0) * CK, have = min(CK, n_req - first);
  if (first < 0 || have <= 0 || n_req < from) return false;
  const size_t t0 = (size_t)(t_req + first);
  const int kh = h / (H / G);
  {
    float4 in[EACH][3], bias[EACH];
    const float strong = tid < have ? pbeta[(t0 + tid) * H + h] : 0.f, rate = -expf(a_log[h]);
#pragma unroll
    for (int x = 0; x < EACH; ++x) {
      const int e = tid + x * GCR_THREADS, t = e / (DMAX / 4), c = e % (DMAX / 4) * 4;
      in[x][0] = in[x][1] = in[x][2] = bias[x] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < have && c < d) {
        const size_t at = ((t0 + t) * G + kh) * d + c;
        in[x][0] = __ldg(reinterpret_cast<const float4*>(pq + at));
        in[x][1] = __ldg(reinterpret_cast<const float4*>(pk + at));
        const float *a = araw + ((t0 + t) * H + h) * d + c, *b = dt_bias + (size_t)h * d + c;      // (any alignment)
        in[x][2] = make_float4(__ldg(a), __ldg(a + 1), __ldg(a + 2), __ldg(a + 3));
        bias[x] = make_float4(__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3));
      }
    }
    if (tid < CK) strength[tid] = strong;
    auto decay = [&](float a, float b) { return expf(rate * rec_softplus(a + b)); };
#pragma unroll
    for (int x = 0; x < EACH; ++x) {
      const int e = tid + x * GCR_THREADS, t = e / (DMAX / 4), c = e % (DMAX / 4) * 4;
      if (t >= CK) continue;
      float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
      if (t < have && c < d)
        w = make_float4(decay(in[x][2].x, bias[x].x), decay(in[x][2].y, bias[x].y), decay(in[x][2].z, bias[x].z), decay(in[x][2].w, bias[x].w));
      *reinterpret_cast<float4*>(&q[t][c]) = in[x][0];
      *reinterpret_cast<float4*>(&k[t][c]) = in[x][1];
      *reinterpret_cast<float4*>(&g[t][c]) = w;
    }
  }
  __syncthreads();
  {
    struct alignas(4 * PER) Piece { float x[PER]; };
    auto piece = [&](const float* row) { return *reinterpret_cast<const Piece*>(row + PER * lane); };
    Piece kj = piece(k[warp]);
    for (int step = 0; step <= CK; ++step) {      // token `warp` through the tokens from it on, then token 15 - warp
      const bool second = step >= CK - warp;
      const int j = second ? CK - 1 - warp : warp, i = second ? step - 1 : warp + step;
      if (step == CK - warp) kj = piece(k[j]);
      const Piece qi = piece(q[i]), ki = piece(k[i]), w = piece(g[i]);
      float a = 0.f, b = 0.f;                     // q_i . k_j, k_i . k_j
#pragma unroll
      for (int m = 0; m < PER; ++m) {
        if (i > j) kj.x[m] *= w.x[m];
        a = fmaf(qi.x[m], kj.x[m], a);
        b = fmaf(ki.x[m], kj.x[m], b);
      }
      const bool high = lane & 16;
      float s = (high ? b : a) + __shfl_xor_sync(0xffffffffu, high ? a : b, 16);
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
      if ((lane & 15) == 0) sums[high][i][j] = s;
    }
  }
  // The values that this warp needs below are on their way.
  float v[8];
  auto fetch = [&](int group) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int t = ck_token(lane, e), col = 16 * group + ck_channel(lane, e);
      v[e] = t < have && col < dv ? __ldg(pv + ((t0 + t) * H + h) * dv + col) : 0.f;
    }
  };
  if (16 * warp < dv) fetch(warp);
  __syncthreads();
  // The rows with their decays: q and -k from the chunk's start, k to its end (in g's place). Beside that the system.
  if (tid < DMAX) {
    float up = 1.f, down = 1.f, to_end[CK];
#pragma unroll
    for (int t = CK - 1; t >= 0; --t) {
      to_end[t] = k[t][tid] * down;
      down *= g[t][tid];
    }
#pragma unroll
    for (int t = 0; t < CK; ++t) {
      up *= g[t][tid];
      q[t][tid] *= up;
      k[t][tid] *= -up;
      g[t][tid] = to_end[t];
    }
    tile[ck_rows(CK_SYSTEM, DMAX) + tid] = up;
    if (tid == 0) tile[ck_flag(DMAX)] = __int_as_float(CAREFUL);
  } else if (warp == 4 && lane < CK) {
#pragma unroll
    for (int i = 0; i < CK; ++i) sums[1][i][lane] *= strength[i];      // (each lane its own column)
    __syncwarp(0xffffu);
    ck_solve<CAREFUL>(&sums[1][0][0], GS, 1.f, lane, strength[lane], T);
  } else if (warp > 4) {
    for (int e = tid - 160; e < CK * CK; e += GCR_THREADS - 160) ck_set<CAREFUL>(Q, e / CK, e % CK, e % CK <= e / CK ? sums[0][e / CK][e % CK] : 0.f);
  }
  __syncthreads();
  for (int c0 = 16 * warp; c0 < DMAX; c0 += 16 * (GCR_THREADS / 32)) {
    uint32_t a[3][4];
    float x[8], f[8], b[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int t = ck_token(lane, e), c = c0 + ck_channel(lane, e);
      x[e] = k[t][c];
      f[e] = q[t][c];
      b[e] = g[t][c];
    }
    ck_system_rows<CAREFUL>(tile, CK_W, ROW, c0, lane, T, Q, x, f, look);
    ck_operand_of<CAREFUL>(f, a, look);
    ck_put(tile, CK_F, ROW, c0, lane, a);
    ck_operand_of<CAREFUL>(b, a, look);
    ck_put(tile, CK_B, ROW, c0, lane, a);
  }
  ck_tile_written();
  for (int group = warp; 16 * group < dv; group += GCR_THREADS / 32) {
    if (group != warp) fetch(group);
    float y[8], o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = o[e] = 0.f;
    ck_apply<CAREFUL>(T, v, lane, y, look);
    ck_apply<CAREFUL>(Q, y, lane, o, look);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int t = ck_token(lane, e), col = 16 * group + ck_channel(lane, e);
      if (t < have && col < dv) {
        p.u[((t0 + t) * H + h) * dv + col] = y[e];
        p.g_out[((t0 + t) * H + h) * dv + col] = o[e];
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    ck_tile_leaves(p.tiles + ((size_t)place * H + h) * ck_tile(CK_SYSTEM, DMAX), tile, ck_tile(CK_SYSTEM, DMAX));
    ck_tile_left();
  }
  return !CAREFUL && look.found();
}
template <int DMAX>
__device__ __noinline__ void gdr_channel_rows_carefully(const GcrArgs& p, float* tile, GcrShared& sh) {
  ck_tile_again();
  gdr_channel_rows<DMAX, true>(p, tile, sh);
}
template <int DMAX>
__global__ void __launch_bounds__(GCR_THREADS, 3) gdr_channel_rows_kernel(const __grid_constant__ GcrArgs p) {
  extern __shared__ __align__(128) float gcr_raw[];
  __shared__ GcrShared sh;
  if (__syncthreads_or(gdr_channel_rows<DMAX, false>(p, gcr_raw, sh))) gdr_channel_rows_carefully<DMAX>(p, gcr_raw, sh);
}
template <int DMAX>
static int launch_channel_rows(dim3 grid, cudaStream_t stream, const GcrArgs& p) {
  constexpr size_t smem = gcr_smem(DMAX);
  cudaError_t e = cudaFuncSetAttribute(gdr_channel_rows_kernel<DMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return llmrs_fail("gated_delta: shared memory %zu: %s", smem, cudaGetErrorString(e));
  gdr_channel_rows_kernel<DMAX><<<grid, GCR_THREADS, smem, stream>>>(p);
  return llmrs_launch_status("gated_delta (chunks)");
}

// ---- the recurrence in chunks ------------------------------------------------------------------------------------
constexpr int GC_C = 32, GC_W = 16, GC_THREADS = 128, GC_TST = GC_C + 4;
// A chunk's tables in the workspace: T [C][C], P [C][C], e^{L_t} [C], e^{L_C - L_t} [C].
constexpr int GC_TABLE = 2 * GC_C * GC_C + 2 * GC_C;
// The place of request `req`'s chunk `k`: requests' chunks follow one another; floor(q_start / C) + req leaves every
// request at least ceil(n / C) places.
__device__ __forceinline__ int gc_slot(int q_start, int req, int k) { return q_start / GC_C + req + k; }

__global__ void __launch_bounds__(GC_THREADS)
gdr_chunk_tables_kernel(const float* __restrict__ pq, const float* __restrict__ pk, const float* __restrict__ pbeta,
                        const float* __restrict__ plg, const int* __restrict__ q_start, const int* __restrict__ n_new,
                        float* __restrict__ tables, int G, int H, int d) {
  extern __shared__ float sm[];
  const int req = blockIdx.x, chunk = blockIdx.y, head = blockIdx.z;
  const int n = n_new[req], c0 = chunk * GC_C;
  if (c0 >= n) return;
  const int cn = min(GC_C, n - c0), t0 = q_start[req] + c0, kh = head / (H / G), wq = G * d, st = d + 1;
  float* Ks = sm;                      // [C][d + 1]
  float* Qs = Ks + GC_C * st;          // [C][d + 1]
  float* A = Qs + GC_C * st;           // [C][C + 1]
  float* L = A + GC_C * (GC_C + 1);    // [C]
  float* B = L + GC_C;                 // [C]
  float* out = tables + ((size_t)gc_slot(q_start[req], req, chunk) * H + head) * GC_TABLE;
  for (int e = threadIdx.x; e < GC_C * d; e += GC_THREADS) {
    const int t = e / d, i = e % d;
    Ks[t * st + i] = t < cn ? pk[(size_t)(t0 + t) * wq + (size_t)kh * d + i] : 0.f;
    Qs[t * st + i] = t < cn ? pq[(size_t)(t0 + t) * wq + (size_t)kh * d + i] : 0.f;
  }
  if (threadIdx.x < GC_C) B[threadIdx.x] = threadIdx.x < cn ? pbeta[(size_t)(t0 + threadIdx.x) * H + head] : 0.f;
  if (threadIdx.x == 0) {
    float run = 0.f;
    for (int t = 0; t < GC_C; ++t) {
      if (t < cn) run += plg[(size_t)(t0 + t) * H + head];
      L[t] = run;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < GC_C * GC_C; e += GC_THREADS) {
    const int t = e / GC_C, s_ = e % GC_C;
    float a = 0.f, p = 0.f;
    if (s_ <= t) {
      const float* kt = Ks + t * st;
      const float* qt = Qs + t * st;
      const float* ks = Ks + s_ * st;
      for (int i = 0; i < d; ++i) {
        a = fmaf(kt[i], ks[i], a);
        p = fmaf(qt[i], ks[i], p);
      }
      const float w = expf(L[t] - L[s_]);
      a *= w;
      p *= w;
    }
    A[t * (GC_C + 1) + s_] = s_ < t ? a : 0.f;
    out[GC_C * GC_C + e] = p;
  }
  if (threadIdx.x < GC_C) {
    out[2 * GC_C * GC_C + threadIdx.x] = expf(L[threadIdx.x]);
    out[2 * GC_C * GC_C + GC_C + threadIdx.x] = expf(L[GC_C - 1] - L[threadIdx.x]);
  }
  __syncthreads();
  // T = (I + diag(beta) A)^{-1} diag(beta) by forward substitution: a thread per column.
  if (threadIdx.x < GC_C) {
    const int c = threadIdx.x;
    float col[GC_C];
#pragma unroll
    for (int t = 0; t < GC_C; ++t) {
      float acc = t == c ? 1.0f : 0.f;
#pragma unroll
      for (int s_ = 0; s_ < GC_C; ++s_)
        if (s_ < t) acc = fmaf(-A[t * (GC_C + 1) + s_], col[s_], acc);
      col[t] = t >= c ? B[t] * acc : 0.f;
    }
#pragma unroll
    for (int t = 0; t < GC_C; ++t) out[t * GC_C + c] = col[t];
  }
}

// Shared memory of the chunked recurrence, in floats: two buffers of (K, Q rows [C][d + 4], T, P [C][C + 4], V [C][W],
// e^L, e^{L_C - L}), then the state slice [d][W], V' and U [C][W] each.
__host__ __device__ inline int gc_buffer_floats(int d) { return 2 * GC_C * (d + 4) + 2 * GC_C * GC_TST + GC_C * GC_W + 2 * GC_C; }
__host__ __device__ inline int gc_smem_floats(int d) { return 2 * gc_buffer_floats(d) + d * GC_W + 2 * GC_C * GC_W; }

__global__ void __launch_bounds__(GC_THREADS)
gdr_chunked_kernel(const float* __restrict__ pq, const float* __restrict__ pk, const float* __restrict__ pv,
                   const float* __restrict__ tables, float* __restrict__ state, const int* __restrict__ q_start,
                   const int* __restrict__ n_new, const int* __restrict__ slot_ids, float* __restrict__ o_raw, int G,
                   int H, int d, int dv) {
  extern __shared__ __align__(16) float sm[];
  const int req = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * GC_W;
  const int kh = head / (H / G), tid = threadIdx.x, j = tid & 15, grp = tid >> 4;      // 8 groups of 16 columns' lanes
  const int t_first = q_start[req], n = n_new[req], wq = G * d, wv = H * dv, kst = d + 4;
  const int ncols = min(GC_W, dv - col0);
  const int bufsz = gc_buffer_floats(d);
  float* S0 = sm + 2 * bufsz;            // [d][W]
  float* Vp = S0 + d * GC_W;             // [C][W]
  float* Us = Vp + GC_C * GC_W;          // [C][W]
  float* S_g = state + ((size_t)slot_ids[req] * H + head) * d * dv;
  for (int e = tid; e < d * GC_W; e += GC_THREADS) {
    const int i = e / GC_W, c = e % GC_W;
    S0[e] = c < ncols ? S_g[(size_t)i * dv + col0 + c] : 0.f;
  }
  const int n_chunks = (n + GC_C - 1) / GC_C;
  auto load = [&](int it) {
    float* b = sm + (it & 1) * bufsz;
    float* Ks = b;
    float* Qs = Ks + GC_C * kst;
    float* Ts = Qs + GC_C * kst;
    float* Ps = Ts + GC_C * GC_TST;
    float* Vs = Ps + GC_C * GC_TST;
    float* Gs = Vs + GC_C * GC_W;        // e^L [C], then e^{L_C - L} [C]
    const int c0 = it * GC_C, cn = min(GC_C, n - c0), per_row = d / 4;
    for (int e = tid; e < 2 * GC_C * per_row; e += GC_THREADS) {
      const int a = e / (GC_C * per_row), rem = e % (GC_C * per_row), t = rem / per_row, piece = rem % per_row;
      const bool valid = t < cn;
      const float* src = (a == 0 ? pk : pq) + (valid ? (size_t)(t_first + c0 + t) * wq + (size_t)kh * d + piece * 4 : 0);
      cp_async_16((a == 0 ? Ks : Qs) + t * kst + piece * 4, src, valid ? 16 : 0);
    }
    const float* tb = tables + ((size_t)gc_slot(t_first, req, it) * H + head) * GC_TABLE;
    for (int e = tid; e < 2 * GC_C * (GC_C / 4); e += GC_THREADS) {
      const int a = e / (GC_C * (GC_C / 4)), rem = e % (GC_C * (GC_C / 4)), t = rem / (GC_C / 4), piece = rem % (GC_C / 4);
      cp_async_16((a == 0 ? Ts : Ps) + t * GC_TST + piece * 4, tb + a * GC_C * GC_C + t * GC_C + piece * 4, 16);
    }
    for (int e = tid; e < GC_C * (GC_W / 4); e += GC_THREADS) {
      const int t = e / (GC_W / 4), piece = e % (GC_W / 4);
      const bool valid = t < cn && piece * 4 < ncols;      // dv is a multiple of 4: a piece lies wholly inside or outside
      const float* src = pv + (valid ? (size_t)(t_first + c0 + t) * wv + (size_t)head * dv + col0 + piece * 4 : 0);
      cp_async_16(Vs + t * GC_W + piece * 4, src, valid ? 16 : 0);
    }
    for (int e = tid; e < 2 * GC_C / 4; e += GC_THREADS) cp_async_16(Gs + e * 4, tb + 2 * GC_C * GC_C + e * 4, 16);
    cp_async_commit();
  };
  if (n_chunks > 0) load(0);
  for (int it = 0; it < n_chunks; ++it) {
    if (it + 1 < n_chunks) {
      load(it + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* b = sm + (it & 1) * bufsz;
    const float* Ks = b;
    const float* Qs = Ks + GC_C * kst;
    const float* Ts = Qs + GC_C * kst;
    const float* Ps = Ts + GC_C * GC_TST;
    const float* Vs = Ps + GC_C * GC_TST;
    const float* Gs = Vs + GC_C * GC_W;
    const float* Ds = Gs + GC_C;
    const int c0 = it * GC_C, cn = min(GC_C, n - c0);
    // This thread's four tokens grp, grp + 8, grp + 16, grp + 24 of column j.
    float x[4] = {0.f, 0.f, 0.f, 0.f}, qs[4] = {0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < d; i += 4) {
      const float s0 = S0[(i + 0) * GC_W + j], s1 = S0[(i + 1) * GC_W + j], s2 = S0[(i + 2) * GC_W + j],
                  s3 = S0[(i + 3) * GC_W + j];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float4 k4 = *reinterpret_cast<const float4*>(Ks + (grp + 8 * m) * kst + i);
        const float4 q4 = *reinterpret_cast<const float4*>(Qs + (grp + 8 * m) * kst + i);
        x[m] = fmaf(k4.w, s3, fmaf(k4.z, s2, fmaf(k4.y, s1, fmaf(k4.x, s0, x[m]))));
        qs[m] = fmaf(q4.w, s3, fmaf(q4.z, s2, fmaf(q4.y, s1, fmaf(q4.x, s0, qs[m]))));
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int t = grp + 8 * m;
      Vp[t * GC_W + j] = Vs[t * GC_W + j] - Gs[t] * x[m];      // V - e^L (K S_0)
    }
    __syncthreads();
    float u[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s_ = 0; s_ < GC_C; s_ += 4) {
      const float v0 = Vp[(s_ + 0) * GC_W + j], v1 = Vp[(s_ + 1) * GC_W + j], v2 = Vp[(s_ + 2) * GC_W + j],
                  v3 = Vp[(s_ + 3) * GC_W + j];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float4 t4 = *reinterpret_cast<const float4*>(Ts + (grp + 8 * m) * GC_TST + s_);
        u[m] = fmaf(t4.w, v3, fmaf(t4.z, v2, fmaf(t4.y, v1, fmaf(t4.x, v0, u[m]))));
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) Us[(grp + 8 * m) * GC_W + j] = u[m];
    __syncthreads();
    float o[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) o[m] = Gs[grp + 8 * m] * qs[m];
    for (int s_ = 0; s_ < GC_C; s_ += 4) {
      const float u0 = Us[(s_ + 0) * GC_W + j], u1 = Us[(s_ + 1) * GC_W + j], u2 = Us[(s_ + 2) * GC_W + j],
                  u3 = Us[(s_ + 3) * GC_W + j];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float4 p4 = *reinterpret_cast<const float4*>(Ps + (grp + 8 * m) * GC_TST + s_);
        o[m] = fmaf(p4.w, u3, fmaf(p4.z, u2, fmaf(p4.y, u1, fmaf(p4.x, u0, o[m]))));
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int t = grp + 8 * m;
      if (t < cn && j < ncols) o_raw[(size_t)(t_first + c0 + t) * wv + (size_t)head * dv + col0 + j] = o[m];
    }
    // The new state: this thread's key channels [i_lo, i_hi) of column j.
    const int per = ((d + 7) / 8 + 3) & ~3, i_lo = min(grp * per, d), i_hi = min(i_lo + per, d);
    float acc[32];
#pragma unroll
    for (int a = 0; a < 32; ++a) acc[a] = 0.f;
    for (int t = 0; t < GC_C; ++t) {
      const float du = Ds[t] * Us[t * GC_W + j];
#pragma unroll
      for (int a = 0; a < 32; a += 4) {
        if (i_lo + a < i_hi) {
          const float4 k4 = *reinterpret_cast<const float4*>(Ks + t * kst + i_lo + a);
          acc[a] = fmaf(k4.x, du, acc[a]);
          acc[a + 1] = fmaf(k4.y, du, acc[a + 1]);
          acc[a + 2] = fmaf(k4.z, du, acc[a + 2]);
          acc[a + 3] = fmaf(k4.w, du, acc[a + 3]);
        }
      }
    }
    __syncthreads();      // every thread has read the old state
    const float gc = Gs[GC_C - 1];
#pragma unroll
    for (int a = 0; a < 32; ++a)
      if (i_lo + a < i_hi) S0[(i_lo + a) * GC_W + j] = fmaf(gc, S0[(i_lo + a) * GC_W + j], acc[a]);
    // (the next turn's first barrier makes the new state visible; its loads go into the other buffer)
  }
  __syncthreads();
  for (int e = tid; e < d * GC_W; e += GC_THREADS) {
    const int i = e / GC_W, c = e % GC_W;
    if (c < ncols) S_g[(size_t)i * dv + col0 + c] = S0[e];
  }
}

// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * weight[:] * act(gate[t, h, :]), act SiLU or (gate_sigmoid)
// the sigmoid; a warp per (t, h).
template <typename TA>
__global__ void gdr_out_kernel(const float* __restrict__ o_raw, const TA* __restrict__ gate, long long gate_stride,
                               const float* __restrict__ norm_w, TA* __restrict__ out, long long out_stride,
                               int n_rows, int H, int dv, float eps, float out_scale, int gate_sigmoid) {
  const int r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= n_rows) return;
  const int t = r / H, h = r % H;
  const float* o = o_raw + (size_t)t * H * dv + (size_t)h * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss = fmaf(o[i], o[i], ss);
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + eps) * out_scale;
  for (int i = lane; i < dv; i += 32) {
    const float gr = to_float(gate[(size_t)t * gate_stride + (size_t)h * dv + i]);
    const float gt = gate_sigmoid ? rec_sigmoid(gr) : rec_silu(gr);
    out[(size_t)t * out_stride + (size_t)h * dv + i] = from_float<TA>(o[i] * inv * norm_w[i] * gt);
  }
}

static int launch_chunked(const float* pq, const float* pk, const float* pv, const float* pbeta, const float* plg,
                          float* tables, float* state, const int* q_start, const int* n_new, const int* slot_ids,
                          float* o_raw, int n_requests, int max_chunks, int G, int H, int d, int dv,
                          cudaStream_t stream) {
  const size_t smem_t = ((size_t)2 * GC_C * (d + 1) + GC_C * (GC_C + 1) + 2 * GC_C) * sizeof(float);
  const size_t smem_c = (size_t)gc_smem_floats(d) * sizeof(float);
  static size_t configured_t = 48 * 1024, configured_c = 48 * 1024;
  if (smem_t > configured_t) {
    cudaError_t e = cudaFuncSetAttribute(gdr_chunk_tables_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_t);
    if (e != cudaSuccess) return llmrs_fail("gated_delta: shared memory %zu: %s", smem_t, cudaGetErrorString(e));
    configured_t = smem_t;
  }
  if (smem_c > configured_c) {
    cudaError_t e = cudaFuncSetAttribute(gdr_chunked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c);
    if (e != cudaSuccess) return llmrs_fail("gated_delta: shared memory %zu: %s", smem_c, cudaGetErrorString(e));
    configured_c = smem_c;
  }
  LLMRS_REQUIRE(max_chunks <= 65535, "gated_delta: a portion of %d chunks is too long", max_chunks);
  gdr_chunk_tables_kernel<<<dim3(n_requests, max_chunks, H), GC_THREADS, smem_t, stream>>>(pq, pk, pbeta, plg, q_start,
                                                                                           n_new, tables, G, H, d);
  int rc = llmrs_launch_status("gated_delta (chunk tables)");
  if (rc != 0) return rc;
  gdr_chunked_kernel<<<dim3(n_requests, H, (dv + GC_W - 1) / GC_W), GC_THREADS, smem_c, stream>>>(
      pq, pk, pv, tables, state, q_start, n_new, slot_ids, o_raw, G, H, d, dv);
  return llmrs_launch_status("gated_delta (chunked recurrence)");
}

struct TurnRows {      // what gdr_turns_kernel leaves in the workspace
  float *pq, *pk, *kb, *pv, *w, *tables, *pbeta, *pg;
};
template <typename TA>
static int launch_turns(const TA* x, long long x_stride, const float* taps, const float* ba, const TA* b, long long b_stride,
                        const float* araw, const float* a_log, const float* dt_bias, const float* conv_state, const TurnRows& r,
                        const int* q_start, const int* n_new, const int* slot_ids, int n_tokens, int n_requests, int G, int H,
                        int d, int dv, int K, float key_eps, float q_scale, int from, bool chunks, cudaStream_t stream) {
  auto rows_of_four = [](const void* p, size_t size, long long stride) { return ((uintptr_t)p & (4 * size - 1)) == 0 && stride % 4 == 0; };
  const bool vec = d % 4 == 0 && H * dv % 4 == 0 && rows_of_four(x, sizeof(TA), x_stride) && rows_of_four(conv_state, 4, 4) &&
                   rows_of_four(araw, 4, 4);
  const bool taps4 = K == 4 && ((uintptr_t)taps & 15) == 0;
  const int cpl = d <= 128 ? 4 : 8, units = G + (H * dv + 32 * cpl - 1) / (32 * cpl);
  LLMRS_REQUIRE((units + 3) / 4 <= 65535, "gated_delta: too many heads");
  const dim3 grid((unsigned)walk_places(n_tokens, n_requests), (units + 3) / 4);
#define LLMRS_GD_TURNS(CPL, CH, CHUNKS)                                                                                       \
  gdr_turns_kernel<TA, CPL, CH, CHUNKS><<<grid, 128, 0, stream>>>(x, x_stride, taps, ba, b, b_stride, araw, a_log, dt_bias, conv_state, \
                                                          q_start, n_new, slot_ids, r.pq, r.pk, r.kb, r.pv, r.w, r.tables, r.pbeta, r.pg, \
                                                          n_requests, G, H, d, dv, K, key_eps, q_scale, vec, taps4, from)
  if (araw && chunks) LLMRS_GD_TURNS(4, true, true);
  else if (chunks) LLMRS_GD_TURNS(4, false, true);
  else if (araw && cpl == 4) LLMRS_GD_TURNS(4, true, false);
  else if (araw) LLMRS_GD_TURNS(8, true, false);
  else if (cpl == 4) LLMRS_GD_TURNS(4, false, false);
  else LLMRS_GD_TURNS(8, false, false);
#undef LLMRS_GD_TURNS
  return llmrs_launch_status("gated_delta (turns)");
}

static int launch_turn_walk(bool channel, const TurnRows& r, float* state, const int* q_start, const int* n_new,
                            const int* slot_ids, float* o_raw, int n_requests, int G, int H, int d, int dv, int from,
                            cudaStream_t stream) {
  WalkArgs a = {};
  a.q = r.pq; a.k = r.pk; a.kb = r.kb; a.w = r.w;
  a.v = r.pv; a.tables = r.tables; a.state = state; a.o_raw = o_raw;
  a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
  a.n_heads = H; a.d = d; a.dv = dv; a.from = from;
  a.n_groups = channel ? H : G;
  a.q_stride = a.k_stride = a.b_stride = (long long)a.n_groups * d;
  return channel ? launch_state_walk<WALK_CHANNEL>(a, n_requests, dv, stream) : launch_state_walk<WALK_GATED>(a, n_requests, dv, stream);
}

// The chunks' counterpart: pq, pk, pv, pbeta (and pg) hold the rows as gdr_turns_kernel<CHUNKS> left them.
static int launch_chunk_walk(bool channel, const TurnRows& r, float* work, const float* araw, const float* a_log,
                             const float* dt_bias, float* state, const int* q_start, const int* n_new, const int* slot_ids,
                             float* o_raw, int n_tokens, int n_requests, int G, int H, int d, int dv, int from,
                             cudaStream_t stream) {
  float *u = work, *g = u + (size_t)n_tokens * H * dv, *tiles = g + (size_t)n_tokens * H * dv;
  int rc;
  if (channel) {
    LLMRS_REQUIRE(H <= 65535, "gated_delta: too many heads");
    const dim3 grid((unsigned)ck_places(n_tokens, n_requests, from), H);
    const GcrArgs a = {r.pq, r.pk, r.pv, r.pbeta, araw, a_log, dt_bias, q_start, n_new, tiles, u, g, n_requests, G, H, d, dv, from};
    rc = (d <= 64 ? launch_channel_rows<64> : launch_channel_rows<128>)(grid, stream, a);
  } else {
    ChunkRowsArgs a = {};
    a.q = r.pq; a.k = r.pk; a.stride = (long long)G * d; a.v = r.pv; a.decay = r.pg; a.beta = r.pbeta;
    a.q_start = q_start; a.n_new = n_new; a.tiles = tiles; a.u = u; a.g = g;
    a.n_requests = n_requests; a.n_heads = H; a.n_groups = G; a.d = d; a.dv = a.columns = dv; a.from = from;
    rc = launch_ck_rows<CK_SYSTEM>(a, n_tokens, stream);
  }
  if (rc != 0) return rc;
  ChunkArgs a = {};
  a.tiles = tiles; a.u = u; a.g = g; a.state = state; a.o_raw = o_raw;
  a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
  a.n_heads = H; a.d = d; a.dv = a.columns = dv; a.from = from;
  return launch_state_chunks<CK_SYSTEM>(a, n_requests, stream);
}

static int g_gd_chunked = 0;
// 1: portions of 64 tokens and more take the chunked form (off by default: it is not ahead yet, see the file's head).
LLMRS_API void llmrs_gated_delta_chunked(int on) { g_gd_chunked = on; }

// Float32 workspace of the kernels, in floats: prepared q, k, v, beta, g and the raw read-outs; where requests are walked (walk_from as
// below) their coefficients and decays in turns, their rows in chunks.
LLMRS_API long long llmrs_gated_delta_work_floats(int n_tokens, int n_requests, int G, int H, int d, int dv, int channel, int walk_from) {
  const long long prepared = (long long)n_tokens * (2LL * G * d + 2LL * H * dv + (channel ? 1LL * H * d + H : 3LL * H)) + 48;
  const long long form = g_gd_chunked && !channel ? (n_tokens / GC_C + n_requests + 1LL) * H * GC_TABLE : 0;
  if (walk_from <= 0) return prepared + form;
  if (ck_takes(CK_SYSTEM, d, dv)) return prepared + std::max(form, ck_work_floats(CK_SYSTEM, n_tokens, n_requests, walk_from, H, d, dv));
  const long long turns = walk_places(n_tokens, n_requests) * H;
  if (channel) return prepared + 3LL * n_tokens * H * d + turns * (d + walk_table(WALK_CHANNEL));
  return prepared + std::max(form, turns * walk_table(WALK_GATED));
}

// x: [tokens, >= 2 G d + H dv] of `dtype`, rows `x_stride` apart: the q, k and v channels that enter the convolutions;
// gate: [tokens, H dv] rows `gate_stride` apart; taps: float32 [2 G d + H dv, K]; state: float32 [slots, H, d, dv];
// conv_state: float32 [slots, K - 1, 2 G d + H dv]; work: 16-byte aligned; out: [tokens, H dv] rows `out_stride` apart,
// multiplied by `out_scale`. A decay per head: ba float32 [tokens, 2 H] (b, then a), dt_bias [H]. A decay per key channel
// (araw not null; ba unused): b [tokens, H] of `dtype` rows `b_stride` apart, araw float32 [tokens, H d], dt_bias [H d].
// walk_from: requests of at least so many tokens are walked in turns, the others token by token; 0: all of them are.
LLMRS_API int llmrs_gated_delta(const void* x, long long x_stride, const void* gate, long long gate_stride, int dtype,
                                const float* taps, const float* ba, const void* b, long long b_stride, const float* araw,
                                const float* a_log, const float* dt_bias, const float* norm_w, float* state,
                                float* conv_state, const int* token_req, const int* q_start, const int* n_new,
                                const int* slot_ids, float* work, void* out, long long out_stride, int n_tokens,
                                int n_requests, int G, int H, int d, int dv, int K, float key_eps, float q_scale,
                                float norm_eps, float out_scale, int gate_sigmoid, int walk_from, cudaStream_t stream) {
  LLMRS_REQUIRE(n_requests >= 0 && n_tokens >= 0 && G > 0 && H > 0 && d > 0 && dv > 0 && K >= 1, "gated_delta: bad sizes");
  LLMRS_REQUIRE(H % G == 0, "gated_delta: %d value heads are no multiple of %d key heads", H, G);
  LLMRS_REQUIRE(d <= 256, "gated_delta: key heads of at most 256 channels, got %d", d);
  LLMRS_REQUIRE(H <= 65535 && (dv + GD_COLS - 1) / GD_COLS <= 65535, "gated_delta: too many heads or columns");
  LLMRS_REQUIRE(((uintptr_t)work & 15) == 0, "gated_delta: the workspace must be 16-byte aligned");
  LLMRS_REQUIRE(araw ? b != nullptr : ba != nullptr, "gated_delta: no write strengths");
  if (n_requests == 0 || n_tokens == 0) return 0;
  const bool channel = araw != nullptr;
  const int wq = G * d, wv = H * dv, C = 2 * wq + wv;
  LLMRS_REQUIRE((size_t)C * sizeof(float) <= 160 * 1024, "gated_delta: %d convolution channels are too many", C);
  // Every piece starts on a 16-byte boundary (the recurrence copies rows sixteen bytes at a time).
  auto up4 = [](size_t v) { return (v + 3) & ~(size_t)3; };
  float* pq = work;
  float* pk = pq + up4((size_t)n_tokens * wq);
  float* pv = pk + up4((size_t)n_tokens * wq);
  float* pbeta = pv + up4((size_t)n_tokens * wv);
  float* pg = pbeta + up4((size_t)n_tokens * H);
  float* plg = pg + up4((size_t)n_tokens * H * (channel ? d : 1));
  float* o_raw = channel ? plg : plg + up4((size_t)n_tokens * H);
  float* tables = o_raw + up4((size_t)n_tokens * wv);
  // The chunked form where some request may bring 64 tokens or more (what the host knows: tokens and requests) and the
  // rows can be copied sixteen bytes at a time.
  const bool chunked = g_gd_chunked && !channel && n_tokens - n_requests + 1 >= 2 * GC_C && d % 4 == 0 && dv % 4 == 0 &&
                       (size_t)gc_smem_floats(d) * sizeof(float) <= 200 * 1024;
  const int max_chunks = (n_tokens - n_requests + 1 + GC_C - 1) / GC_C;
  const int from = chunked ? 0 : walk_from, below = from > 0 ? from : INT_MAX;
  // The walk's rows with a decay per key channel follow o_raw; its tables lie where the chunked form's would.
  const size_t hd = up4((size_t)n_tokens * H * d);
  float *qf = tables, *kf = qf + hd, *kb = kf + hd, *turn_w = kb + hd;
  const bool sixteens = from > 0 && ck_takes(CK_SYSTEM, d, dv);
  float* chunk_work = tables;
  if (channel) tables = turn_w + up4((size_t)walk_places(n_tokens, n_requests) * H * d);
  const size_t smem = (size_t)C * sizeof(float);
  const int dmax = d <= 32 ? 32 : (d <= 64 ? 64 : (d <= 128 ? 128 : 256));
  dim3 grid(n_requests, H, (dv + GD_COLS - 1) / GD_COLS);
  const int rows = n_tokens * H;
  HeadOutArgs head = {};
  head.o = o_raw; head.gate = gate; head.gate_stride = gate_stride; head.w = norm_w; head.w_shared = 1;
  head.out = out; head.out_stride = out_stride; head.n_tokens = n_tokens; head.n_heads = H; head.dv = dv;
  head.eps = norm_eps; head.out_scale = out_scale; head.silu = !gate_sigmoid;
#define LLMRS_GD_REC(DMAX, LANES, CH)                                                                             \
  do {                                                                                                           \
    if (from > 0)                                                                                                \
      gdr_recurrence_kernel<DMAX, LANES, CH, true><<<grid, GD_COLS * LANES, 0, stream>>>(                        \
          pq, pk, pv, pbeta, pg, state, q_start, n_new, slot_ids, o_raw, G, H, d, dv, below);                    \
    else                                                                                                         \
      gdr_recurrence_kernel<DMAX, LANES, CH, false><<<grid, GD_COLS * LANES, 0, stream>>>(                       \
          pq, pk, pv, pbeta, pg, state, q_start, n_new, slot_ids, o_raw, G, H, d, dv, below);                    \
  } while (0)
#define LLMRS_GD_REC_ALL(CH, LANES)                                                                              \
  do {                                                                                                           \
    if (dmax == 32) LLMRS_GD_REC(32, (LANES < 8 ? LANES : 8), CH);                                               \
    else if (dmax == 64) LLMRS_GD_REC(64, LANES, CH);                                                            \
    else if (dmax == 128) LLMRS_GD_REC(128, LANES, CH);                                                          \
    else LLMRS_GD_REC(256, LANES, CH);                                                                           \
  } while (0)
#define LLMRS_GD_PREPARE(T, CH)                                                                                        \
  do {                                                                                                                 \
    static size_t configured = 48 * 1024;                                                                              \
    if (smem > configured) {                                                                                           \
      cudaError_t e =                                                                                                  \
          cudaFuncSetAttribute(gdr_prepare_kernel<T, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);     \
      if (e != cudaSuccess) return llmrs_fail("gated_delta: shared memory %zu: %s", smem, cudaGetErrorString(e));      \
      configured = smem;                                                                                               \
    }                                                                                                                  \
    gdr_prepare_kernel<T, CH><<<n_tokens, 256, smem, stream>>>(                                                        \
        (const T*)x, x_stride, taps, ba, (const T*)b, b_stride, araw, a_log, dt_bias, conv_state, token_req, q_start,  \
        n_new, slot_ids, pq, pk, pv, pbeta, pg, plg, G, H, d, dv, K, key_eps, q_scale, below);                         \
  } while (0)
  const bool decayed = channel && !sixteens;
  const TurnRows turn_rows = {decayed ? qf : pq, decayed ? kf : pk, kb, pv, turn_w, tables, pbeta, pg};
#define LLMRS_GD_LAUNCH(T)                                                                                             \
  do {                                                                                                                 \
    int rc = 0;                                                                                                        \
    if (from > 0) {                                                                                                    \
      rc = launch_turns<T>((const T*)x, x_stride, taps, ba, (const T*)b, b_stride, araw, a_log, dt_bias, conv_state,   \
                           turn_rows, q_start, n_new, slot_ids, n_tokens, n_requests, G, H, d, dv, K, key_eps,         \
                           q_scale, from, sixteens, stream);                                                           \
      if (rc != 0) return rc;                                                                                          \
    }                                                                                                                  \
    if (from != 1) {                                                                                                   \
      if (channel) LLMRS_GD_PREPARE(T, true);                                                                          \
      else LLMRS_GD_PREPARE(T, false);                                                                                 \
      rc = llmrs_launch_status("gated_delta (prepare)");                                                               \
    }                                                                                                                  \
    if (rc != 0) return rc;                                                                                            \
    rc = launch_short_conv_state((const T*)x, x_stride, conv_state, q_start, n_new, slot_ids, n_requests, C, K, stream); \
    if (rc != 0) return rc;                                                                                            \
    if (chunked) {                                                                                                     \
      rc = launch_chunked(pq, pk, pv, pbeta, plg, tables, state, q_start, n_new, slot_ids, o_raw, n_requests,          \
                          max_chunks, G, H, d, dv, stream);                                                            \
      if (rc != 0) return rc;                                                                                          \
    } else if (sixteens) {                                                                                             \
      rc = launch_chunk_walk(channel, turn_rows, chunk_work, araw, a_log, dt_bias, state, q_start, n_new, slot_ids, o_raw, \
                             n_tokens, n_requests, G, H, d, dv, from, stream);                                         \
      if (rc != 0) return rc;                                                                                          \
    } else if (from > 0) {                                                                                             \
      rc = launch_turn_walk(channel, turn_rows, state, q_start, n_new, slot_ids, o_raw, n_requests, G, H, d, dv, from, \
                            stream);                                                                                   \
      if (rc != 0) return rc;                                                                                          \
    }                                                                                                                  \
    if (chunked || from == 1) {                                                                                        \
    } else if (channel && (long long)grid.x * grid.y * grid.z <= GD_WIDE_MAX_BLOCKS) LLMRS_GD_REC_ALL(true, 16);       \
    else if (channel) LLMRS_GD_REC_ALL(true, 8);                                                                       \
    else LLMRS_GD_REC_ALL(false, LLMRS_GD_LANES);                                                                      \
    rc = llmrs_launch_status("gated_delta (recurrence)");                                                              \
    if (rc != 0) return rc;                                                                                            \
    if (head_out_takes<T>(head)) launch_head_out<T>(head, stream);                                                     \
    else                                                                                                               \
      gdr_out_kernel<T><<<(rows + 3) / 4, 128, 0, stream>>>(o_raw, (const T*)gate, gate_stride, norm_w, (T*)out,       \
                                                            out_stride, rows, H, dv, norm_eps, out_scale, gate_sigmoid); \
  } while (0)
  if (dtype == LLMRS_F32) LLMRS_GD_LAUNCH(float);
  else if (dtype == LLMRS_BF16) LLMRS_GD_LAUNCH(__nv_bfloat16);
  else return llmrs_fail("gated_delta: unknown dtype %d", dtype);
#undef LLMRS_GD_LAUNCH
#undef LLMRS_GD_PREPARE
#undef LLMRS_GD_REC_ALL
#undef LLMRS_GD_REC
  return llmrs_launch_status("gated_delta (norm and gate)");
}
