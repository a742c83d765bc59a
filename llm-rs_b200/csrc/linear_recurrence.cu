// Linear recurrences with a matrix state per head, the common core of gated linear attention and matrix-memory
// recurrent layers:
//
//   S_t = a_t S_(t-1) + (b_t k_t) v_t^T        S: [key channel, value channel], float32, kept per request slot
//   o_t = S_t^T q_t
//
// with a scalar decay a_t and a scalar gain b_t per (token, head). Queries and keys may be shared by groups of heads (head
// h reads group h / (heads / groups)); the gain then multiplies the value instead of the key, and a skip D_h per head adds
// D_h v_t to o_t. A layer with a normaliser also carries
// n_t = a_t n_(t-1) + b_t k_t and divides o_t by max(|n_t . q_t|, floor_t) + den_eps: the normaliser is the state's
// column for a value that is always 1, and is computed as such.
//
// Kernels:
//   gate_scan    exponential gates with a running maximum m (m_t = max(f_t + m_(t-1), i_t), log-space input gate i and
//                forget gate f, both soft-capped): a warp per (request, head) scans the request's tokens of the step,
//                32 at a time (portions of 128 tokens and more: a block each, eight tokens a thread), with the associative form of the (max, +) recurrence, and leaves
//                a_t = exp(f_t + m_(t-1) - m_t), b_t = exp(i_t - m_t), floor_t = exp(-m_t); m is kept per slot;
//   prepare      q, k, v of all tokens widened to float32 (optional SiLU, optional rotation of the first channels of every
//                head of q and k by halves, q and k scaled, k multiplied by its gain);
//   (requests that are walked: the rows of chunks of sixteen tokens, then the walk, state_chunks.cuh; heads that it does not take: the
//   coefficients of turns of four tokens, then the walk, state_walk.cuh)
//   recurrence   of the others: a block per (request, head, 16 value columns) walks the tokens in order; four or eight adjacent lanes
//                share a column, each holding its part of the column's key channels in registers; rows arrive through two
//                shared-memory buffers by 16-byte asynchronous copies. A step of one token and a prompt's portion
//                are the same kernel;
//   output       divides by the normaliser, norms each head (or all heads together) by its root mean square,
//                multiplies by a weight (or none) and by sigmoid(gate) or SiLU(gate), rounds to the activation type.
#include <limits.h>

#include <type_traits>

#include "common.cuh"
#include "head_out.cuh"
#include "mma_util.cuh"
#include "short_conv.cuh"
#include "state_chunks.cuh"

__device__ __forceinline__ float lr_logsigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// ---------------------------------------------------------------------------------
// gate_scan
// ---------------------------------------------------------------------------------
// gates: float32 [tokens, 2 * heads] (row stride given): the input gate's pre-activations, then the forget gate's.
// One head of a request, tokens t0 .. t0 + n - 1, by a warp; *mp: its running maximum.
__device__ __forceinline__ void gate_scan_warp(const float* __restrict__ gates, long long stride, float cap, float* __restrict__ mp,
                                               int t0, int n, int head, float* __restrict__ decay, float* __restrict__ gain,
                                               float* __restrict__ floor_, int n_heads) {
  const int lane = threadIdx.x & 31;
  float m = *mp;
  for (int base = 0; base < n; base += 32) {
    const int t = base + lane;
    const bool live = t < n;
    // A lane without a token is the identity of the recurrence: m_out = max(0 + m_in, -inf).
    float f = 0.f, i = -INFINITY;
    if (live) {
      const float* g = gates + (size_t)(t0 + t) * stride;
      i = cap * tanhf(g[head] / cap);
      f = lr_logsigmoid(cap * tanhf(g[n_heads + head] / cap));
    }
    // Inclusive scan of (F, I) with m_out = max(F + m_in, I); later o earlier = (F_e + F_l, max(F_l + I_e, I_l)).
    float F = f, I = i;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float Fe = __shfl_up_sync(0xffffffffu, F, o), Ie = __shfl_up_sync(0xffffffffu, I, o);
      if (lane >= o) {
        I = fmaxf(F + Ie, I);
        F = Fe + F;
      }
    }
    const float m_t = fmaxf(F + m, I);
    float m_prev = __shfl_up_sync(0xffffffffu, m_t, 1);
    if (lane == 0) m_prev = m;
    if (live) {
      const size_t at = (size_t)(t0 + t) * n_heads + head;
      decay[at] = expf(f + m_prev - m_t);
      gain[at] = expf(i - m_t);
      floor_[at] = expf(-m_t);
    }
    m = __shfl_sync(0xffffffffu, m_t, 31);      // idle lanes carry the last token's value on
  }
  if (lane == 0) *mp = m;
}

__global__ void gate_scan_kernel(const float* __restrict__ gates, long long stride, float cap,
                                 float* __restrict__ m_state, const int* __restrict__ q_start,
                                 const int* __restrict__ n_new, const int* __restrict__ slot_ids,
                                 float* __restrict__ decay, float* __restrict__ gain, float* __restrict__ floor_,
                                 int n_heads) {
  const int req = blockIdx.x, head = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (head >= n_heads) return;
  gate_scan_warp(gates, stride, cap, m_state + (size_t)slot_ids[req] * n_heads + head, q_start[req], n_new[req], head, decay, gain,
                 floor_, n_heads);
}

// The same for steps with a portion of GS_PORTION tokens or more: a block per (request, head), a run of GS_RUN tokens a thread.
// A run's steps compose to one step of the recurrence (F, I); those are scanned over the block, and each thread then walks its
// run from the maximum that it starts with. One warp, 32 tokens at a time, waits for a chain of shuffles and for memory in each
// of its turns: 1,311 tokens of 16 heads 40 us, in runs 8.5. Shorter requests of the step take a warp a head here too, eight
// heads a block, the other blocks of theirs leave at once (257 requests, one of 128 tokens: 9.5 us, 22 with a block a head, 5.6
// by warps alone; 64 requests, one of 512: 6.5, 15.7 by warps alone).
// One portion by a warp / in runs, us: 96 tokens 4.3 / 4.9, 128 5.2 / 5.0, 192 6.9 / 5.1, 512 15.5 / 5.7.
constexpr int GS_RUN = 8, GS_THREADS = 256, GS_PORTION = 128;
__global__ void __launch_bounds__(GS_THREADS)
gate_scan_runs_kernel(const float* __restrict__ gates, long long stride, float cap, float* __restrict__ m_state,
                      const int* __restrict__ q_start, const int* __restrict__ n_new, const int* __restrict__ slot_ids,
                      float* __restrict__ decay, float* __restrict__ gain, float* __restrict__ floor_, int n_heads) {
  __shared__ float s_F[GS_THREADS / 32], s_I[GS_THREADS / 32];
  const int req = blockIdx.x, head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = q_start[req], n = n_new[req];
  if (n < GS_PORTION) {
    const int own = head + warp;
    if (head % (GS_THREADS / 32) == 0 && own < n_heads)
      gate_scan_warp(gates, stride, cap, m_state + (size_t)slot_ids[req] * n_heads + own, t0, n, own, decay, gain, floor_, n_heads);
    return;
  }
  float* mp = m_state + (size_t)slot_ids[req] * n_heads + head;
  float m = *mp;
  __syncthreads();      // every thread has the old maximum before one thread writes the new one
  for (int base = 0; base < n; base += GS_RUN * GS_THREADS) {
    const int first = base + threadIdx.x * GS_RUN;
    float f[GS_RUN], i[GS_RUN], F = 0.f, I = -INFINITY;
#pragma unroll
    for (int e = 0; e < GS_RUN; ++e) {      // a token that is not there is the identity: m_out = max(0 + m_in, -inf)
      const float* g = gates + (size_t)(t0 + first + e) * stride + head;
      i[e] = first + e < n ? g[0] : 0.f;
      f[e] = first + e < n ? g[n_heads] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < GS_RUN; ++e) {
      const bool live = first + e < n;
      i[e] = live ? cap * tanhf(i[e] / cap) : -INFINITY;
      f[e] = live ? lr_logsigmoid(cap * tanhf(f[e] / cap)) : 0.f;
      I = fmaxf(f[e] + I, i[e]);
      F += f[e];
    }
    // Inclusive scan of (F, I); later o earlier = (F_e + F_l, max(F_l + I_e, I_l)).
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float Fe = __shfl_up_sync(0xffffffffu, F, o), Ie = __shfl_up_sync(0xffffffffu, I, o);
      if (lane >= o) {
        I = fmaxf(F + Ie, I);
        F = Fe + F;
      }
    }
    if (lane == 31) {
      s_F[warp] = F;
      s_I[warp] = I;
    }
    const float Fx = __shfl_up_sync(0xffffffffu, F, 1), Ix = __shfl_up_sync(0xffffffffu, I, 1);
    __syncthreads();
    float at_warp = m;      // the maximum that this warp's tokens start with; m: the one after the block's tokens
#pragma unroll
    for (int w = 0; w < GS_THREADS / 32; ++w) {
      if (w == warp) at_warp = m;
      m = fmaxf(s_F[w] + m, s_I[w]);
    }
    float m_prev = lane ? fmaxf(Fx + at_warp, Ix) : at_warp;
#pragma unroll
    for (int e = 0; e < GS_RUN; ++e) {
      if (first + e < n) {
        const float m_t = fmaxf(f[e] + m_prev, i[e]);
        const size_t at = (size_t)(t0 + first + e) * n_heads + head;
        decay[at] = expf(f[e] + m_prev - m_t);
        gain[at] = expf(i[e] - m_t);
        floor_[at] = expf(-m_t);
        m_prev = m_t;
        if (first + e == n - 1) *mp = m_t;
      }
    }
    __syncthreads();      // the runs' steps have been read
  }
}

// longest: no request of the step brings more tokens (it chooses the kernel, not the numbers).
LLMRS_API int llmrs_gate_scan(const float* gates, long long stride, float cap, float* m_state, const int* q_start,
                              const int* n_new, const int* slot_ids, float* decay, float* gain, float* floor_,
                              int longest, int n_requests, int n_heads, cudaStream_t stream) {
  LLMRS_REQUIRE(n_requests >= 0 && n_heads > 0 && cap > 0.f, "gate_scan: bad arguments");
  if (n_requests == 0) return 0;
  if (longest >= GS_PORTION && n_heads <= 65535) {
    gate_scan_runs_kernel<<<dim3(n_requests, n_heads), GS_THREADS, 0, stream>>>(gates, stride, cap, m_state, q_start, n_new,
                                                                                slot_ids, decay, gain, floor_, n_heads);
    return llmrs_launch_status("gate_scan");
  }
  const int warps = n_heads < 4 ? n_heads : 4;
  dim3 grid(n_requests, (n_heads + warps - 1) / warps);
  gate_scan_kernel<<<grid, warps * 32, 0, stream>>>(gates, stride, cap, m_state, q_start, n_new, slot_ids, decay, gain,
                                                    floor_, n_heads);
  return llmrs_launch_status("gate_scan");
}

// ---------------------------------------------------------------------------------
// prepare: float32 planes Q [tokens, heads * dk], K [tokens, heads * dk], V [tokens, heads * dv]
// ---------------------------------------------------------------------------------
// rot_dims > 0: channel i < rot_dims / 2 of every head of q and k is paired with channel i + rot_dims / 2 and the pair
// turned by position * inv_freq[i] (angles in double, after the activation), the other channels pass.
template <typename TA>
__global__ void lr_prepare_kernel(const TA* __restrict__ q, const TA* __restrict__ k, const TA* __restrict__ v,
                                  long long q_stride, long long k_stride, long long v_stride,
                                  const float* __restrict__ gain, const double* __restrict__ inv_freq,
                                  const int* __restrict__ positions, int rot_dims, float* __restrict__ Q,
                                  float* __restrict__ K, float* __restrict__ V, int n_heads, int dk, int dv, int act,
                                  float q_scale, float k_scale) {
  extern __shared__ float cs[];      // [rot_dims / 2][2]
  const int t = blockIdx.x, half = rot_dims / 2;
  const int wk = n_heads * dk, wv = n_heads * dv;
  if (half > 0) {
    const double pos = (double)positions[t];
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
      double s, c;
      sincos(pos * inv_freq[i], &s, &c);
      cs[2 * i] = (float)c;
      cs[2 * i + 1] = (float)s;
    }
    __syncthreads();
  }
  auto at = [&](const TA* row, int c) {
    const float x = to_float(row[c]);
    return act ? x * rec_sigmoid(x) : x;
  };
  auto turned = [&](const TA* row, int c, int i) {
    const float a = at(row, c);
    if (i >= rot_dims) return a;
    const int j = i < half ? i : i - half;
    const float b = at(row, i < half ? c + half : c - half);
    return i < half ? a * cs[2 * j] - b * cs[2 * j + 1] : a * cs[2 * j] + b * cs[2 * j + 1];
  };
  const TA* qr = q + (size_t)t * q_stride;
  const TA* kr = k + (size_t)t * k_stride;
  for (int c = threadIdx.x; c < wk; c += blockDim.x) {
    const int h = c / dk, i = c - h * dk;
    Q[(size_t)t * wk + c] = turned(qr, c, i) * q_scale;
    const float kv = turned(kr, c, i) * k_scale;
    K[(size_t)t * wk + c] = gain ? kv * gain[(size_t)t * n_heads + h] : kv;
  }
  for (int c = threadIdx.x; c < wv; c += blockDim.x) V[(size_t)t * wv + c] = at(v + (size_t)t * v_stride, c);
}

// The same without a rotation, for rows whose pieces of eight channels (four of float32) can be loaded sixteen bytes at a time.
// Bound by memory: 1,793 tokens of 16 heads of 128, a channel a load -> this: 23.4 -> 12.7 us.
template <typename TA>
__global__ void __launch_bounds__(256)
lr_prepare_wide_kernel(const TA* __restrict__ q, const TA* __restrict__ k, const TA* __restrict__ v, long long q_stride,
                       long long k_stride, long long v_stride, const float* __restrict__ gain, float* __restrict__ Q,
                       float* __restrict__ K, float* __restrict__ V, int n_tokens, int n_heads, int dk, int dv, int act,
                       float q_scale, float k_scale) {
  constexpr int N = 16 / sizeof(TA);
  struct alignas(16) Piece { TA x[N]; };
  const int wk = n_heads * dk, wv = n_heads * dv, pk = wk / N, pieces = 2 * pk + wv / N;
  const long long id = (long long)blockIdx.x * 256 + threadIdx.x;
  if (id >= (long long)n_tokens * pieces) return;
  const int t = (int)(id / pieces), p = (int)(id - (long long)t * pieces);
  const int which = p < pk ? 0 : (p < 2 * pk ? 1 : 2), c = (p - which * pk) * N;
  const TA* from = which == 0 ? q + (size_t)t * q_stride : (which == 1 ? k + (size_t)t * k_stride : v + (size_t)t * v_stride);
  float* to = which == 0 ? Q + (size_t)t * wk : (which == 1 ? K + (size_t)t * wk : V + (size_t)t * wv);
  const Piece in = *reinterpret_cast<const Piece*>(from + c);
  float scale = which == 0 ? q_scale : (which == 1 ? k_scale : 1.0f), own = 1.0f;
  if (which == 1 && gain) own = gain[(size_t)t * n_heads + c / dk];
  float y[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    const float x = to_float(in.x[e]);
    y[e] = (act ? x * rec_sigmoid(x) : x) * scale * own;
  }
#pragma unroll
  for (int e = 0; e < N; e += 4) *reinterpret_cast<float4*>(to + c + e) = make_float4(y[e], y[e + 1], y[e + 2], y[e + 3]);
}

// ---------------------------------------------------------------------------------
// recurrence
// ---------------------------------------------------------------------------------
constexpr int LR_COLS = 16;

// LR_LANES adjacent lanes share a column: 4 for heads of up to 64 key channels, 8 above (16 and 32 channels per lane
// instead of 32 and 64: shorter chains of dependent sums per token, and twice the warps on an SM that holds few blocks).
// SOME: only requests of fewer than `below` tokens, the others are walked in turns. (A template: with the test in it a decode step
// of 48 requests of Mamba-2 took 84 us instead of 79.)
template <int DMAX, int LR_LANES, bool SOME>
__global__ void __launch_bounds__(LR_COLS * LR_LANES)
linear_recurrence_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                         const float* __restrict__ decay, const float* __restrict__ head_decay,
                         const float* __restrict__ v_gain, const float* __restrict__ skip, float* __restrict__ S_all, float* __restrict__ N_all, const int* __restrict__ q_start,
                         const int* __restrict__ n_new, const int* __restrict__ slot_ids, float* __restrict__ o_raw,
                         float* __restrict__ nq, int n_heads, int n_groups, int dk, int dv, int below) {
  constexpr int CHUNK = DMAX >= 256 ? 8 : 16;
  constexpr int LR_THREADS = LR_COLS * LR_LANES;
  constexpr int IPL = DMAX / LR_LANES;             // key channels per lane
  __shared__ __align__(16) float s_q[2][CHUNK][DMAX];      // channels >= dk stay 0
  __shared__ __align__(16) float s_k[2][CHUNK][DMAX];
  __shared__ float s_v[2][CHUNK][LR_COLS];
  __shared__ float s_a[2][CHUNK], s_b[2][CHUNK];      // decay, and the gain on the value
  const int req = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * LR_COLS;
  const int tid = threadIdx.x;
  const int col = col0 + tid / LR_LANES, part = tid % LR_LANES;
  // A lane's channels come in groups of four, the groups of a column's lanes interleaved: register 4 g + e holds
  // channel g * 4 * LR_LANES + part * 4 + e, so that the lanes' 16-byte reads of a token's row lie side by side in
  // shared memory (a lane with one run of channels met its neighbours in the same banks).
  auto channel = [&](int i) { return (i >> 2) * 4 * LR_LANES + part * 4 + (i & 3); };
  const int n_cols = dv + (N_all != nullptr ? 1 : 0);      // the normaliser is one more column, whose value is 1
  const bool live = col < n_cols, is_norm = col == dv;
  const int t0 = q_start[req], n = n_new[req];
  if (SOME && n >= below) return;
  const int wk = n_groups * dk, wv = n_heads * dv, group = head / (n_heads / n_groups);
  const size_t slot = (size_t)slot_ids[req];
  float* S_g = S_all + (slot * n_heads + head) * (size_t)dk * dv;
  float* N_g = N_all ? N_all + (slot * n_heads + head) * (size_t)dk : nullptr;
  float S[IPL];
#pragma unroll
  for (int i = 0; i < IPL; ++i) {
    S[i] = 0.f;
    if (live && channel(i) < dk) S[i] = is_norm ? N_g[channel(i)] : S_g[(size_t)channel(i) * dv + col];
  }
  for (int e = tid; e < 2 * CHUNK * DMAX; e += LR_THREADS) {
    (&s_q[0][0][0])[e] = 0.f;
    (&s_k[0][0][0])[e] = 0.f;
  }
  __syncthreads();
  const bool wide = dk % 4 == 0;
  const float a_head = head_decay ? head_decay[head] : 1.0f, d_head = skip ? skip[head] : 0.f;
  auto load_chunk = [&](int buf, int c0) {
    const int cn = min(CHUNK, n - c0);
    if (wide) {
      const int per_row = dk / 4;
      for (int e = tid; e < 2 * cn * per_row; e += LR_THREADS) {
        const int which = e / (cn * per_row), rem = e % (cn * per_row), tt = rem / per_row, piece = rem % per_row;
        const size_t src = (size_t)(t0 + c0 + tt) * wk + (size_t)group * dk + piece * 4;
        cp_async_16(which ? &s_k[buf][tt][piece * 4] : &s_q[buf][tt][piece * 4], (which ? K : Q) + src, 16);
      }
    } else {
      for (int e = tid; e < 2 * cn * dk; e += LR_THREADS) {
        const int which = e / (cn * dk), rem = e % (cn * dk), tt = rem / dk, i = rem % dk;
        const size_t src = (size_t)(t0 + c0 + tt) * wk + (size_t)group * dk + i;
        (which ? s_k : s_q)[buf][tt][i] = (which ? K : Q)[src];
      }
    }
    // Values and decays by 4-byte asynchronous copies too: a plain load would hold the warp for a memory round trip
    // at the top of every chunk, before it starts on the tokens it already has.
    for (int e = tid; e < cn * LR_COLS; e += LR_THREADS) {
      const int tt = e / LR_COLS, c = col0 + e % LR_COLS;
      if (c < dv) cp_async_4(&s_v[buf][tt][e % LR_COLS], V + (size_t)(t0 + c0 + tt) * wv + (size_t)head * dv + c);
      else s_v[buf][tt][e % LR_COLS] = 1.0f;
    }
    for (int tt = tid; tt < cn; tt += LR_THREADS) {
      if (decay) cp_async_4(&s_a[buf][tt], decay + (size_t)(t0 + c0 + tt) * n_heads + head);
      else s_a[buf][tt] = a_head;
      if (v_gain) cp_async_4(&s_b[buf][tt], v_gain + (size_t)(t0 + c0 + tt) * n_heads + head);
      else s_b[buf][tt] = 1.0f;
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
      const float v_in = s_v[buf][tt][tid / LR_LANES], vj = v_in * s_b[buf][tt], a = s_a[buf][tt];
      float os[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < IPL; i += 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(&s_k[buf][tt][i * LR_LANES + part * 4]);
        const float4 q4 = *reinterpret_cast<const float4*>(&s_q[buf][tt][i * LR_LANES + part * 4]);
        S[i] = fmaf(k4.x, vj, a * S[i]);
        S[i + 1] = fmaf(k4.y, vj, a * S[i + 1]);
        S[i + 2] = fmaf(k4.z, vj, a * S[i + 2]);
        S[i + 3] = fmaf(k4.w, vj, a * S[i + 3]);
        os[0] = fmaf(S[i], q4.x, os[0]);
        os[1] = fmaf(S[i + 1], q4.y, os[1]);
        os[2] = fmaf(S[i + 2], q4.z, os[2]);
        os[3] = fmaf(S[i + 3], q4.w, os[3]);
      }
      float o = (os[0] + os[1]) + (os[2] + os[3]);
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      if (LR_LANES == 8) o += __shfl_xor_sync(0xffffffffu, o, 4);
      if (part == 0 && live) {
        if (is_norm) nq[(size_t)(t0 + c0 + tt) * n_heads + head] = o;
        else o_raw[(size_t)(t0 + c0 + tt) * wv + (size_t)head * dv + col] = fmaf(d_head, v_in, o);
      }
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < IPL; ++i)
      if (channel(i) < dk) {
        if (is_norm) N_g[channel(i)] = S[i];
        else S_g[(size_t)channel(i) * dv + col] = S[i];
      }
  }
}

// The recurrence on float32 planes: Q, K [tokens, n_groups * dk], V [tokens, n_heads * dv], each 16-byte aligned; decay
// [tokens, heads] or null (then head_decay [heads], or 1 when that is null too); v_gain [tokens, heads] or null (1)
// multiplies the value that enters the state; skip [heads] or null (0): o += skip * value (without its gain);
// S [slots, heads, dk, dv]; N [slots, heads, dk] or null (no normaliser: nq is not written; with one, v_gain and skip must
// be null); tables: workspace of llmrs_linear_recurrence_table_floats; o_raw float32 [tokens, heads * dv]; nq float32 [tokens,
// heads]. walk_from: requests of at least so many tokens are walked in turns, the others token by token; 0: all of them are.
LLMRS_API int llmrs_linear_recurrence_planes(const float* Q, const float* K, const float* V, const float* decay,
                                             const float* head_decay, const float* v_gain, const float* skip, float* S,
                                             float* N, const int* q_start, const int* n_new, const int* slot_ids,
                                             float* tables, float* o_raw, float* nq, int n_tokens, int n_requests,
                                             int n_heads, int n_groups, int dk, int dv, int walk_from,
                                             cudaStream_t stream) {
  LLMRS_REQUIRE(n_requests >= 0 && n_tokens >= 0 && n_heads > 0 && dk > 0 && dv > 0, "linear_recurrence: bad sizes");
  LLMRS_REQUIRE(n_groups > 0 && n_heads % n_groups == 0, "linear_recurrence: %d heads are no multiple of %d groups",
                n_heads, n_groups);
  LLMRS_REQUIRE(dk <= 256, "linear_recurrence: heads of at most 256 key channels, got %d", dk);
  LLMRS_REQUIRE(n_heads <= 65535 && (dv + 16) / 16 <= 65535, "linear_recurrence: too many heads or columns");
  LLMRS_REQUIRE(N == nullptr || (v_gain == nullptr && skip == nullptr),
                "linear_recurrence: a normaliser goes with gains on the keys");
  LLMRS_REQUIRE((((uintptr_t)Q | (uintptr_t)K) & 15) == 0, "linear_recurrence: planes must be 16-byte aligned");
  if (n_requests == 0 || n_tokens == 0) return 0;
  const int cols = dv + (N != nullptr ? 1 : 0);
  if (walk_from > 0) {
    LLMRS_REQUIRE(((uintptr_t)tables & 15) == 0 && tables != nullptr, "linear_recurrence: no workspace for a portion");
    LLMRS_REQUIRE(((uintptr_t)V & 15) == 0, "linear_recurrence: planes must be 16-byte aligned");
    const long long stride = (long long)n_groups * dk;
    int rc;
    if (ck_takes(CK_LINEAR, dk, dv)) {
      const int columns = ck_columns(dv, N != nullptr);
      ChunkRowsArgs r = {};
      r.q = Q; r.k = K; r.stride = stride; r.v = V; r.decay = decay; r.head_decay = head_decay; r.beta = v_gain; r.skip = skip;
      r.q_start = q_start; r.n_new = n_new; r.n_requests = n_requests; r.n_heads = n_heads; r.n_groups = n_groups;
      r.d = dk; r.dv = dv; r.columns = columns; r.from = walk_from; r.norm = N != nullptr;
      r.u = tables; r.g = r.u + (size_t)n_tokens * n_heads * columns; r.tiles = r.g + (size_t)n_tokens * n_heads * columns;
      rc = launch_ck_rows<CK_LINEAR>(r, n_tokens, stream);
      if (rc != 0) return rc;
      ChunkArgs a = {};
      a.tiles = r.tiles; a.u = r.u; a.g = r.g; a.state = S; a.norm_state = N; a.o_raw = o_raw; a.nq = nq;
      a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
      a.n_heads = n_heads; a.d = dk; a.dv = dv; a.columns = columns; a.from = walk_from;
      rc = launch_state_chunks<CK_LINEAR>(a, n_requests, stream);
    } else {
      rc = launch_walk_tables(Q, K, stride, decay, head_decay, v_gain, q_start, n_new, tables, n_tokens,
                                               n_requests, n_heads, n_groups, dk, walk_from, stream);
      if (rc != 0) return rc;
      WalkArgs a = {};
      a.q = Q; a.k = K; a.q_stride = a.k_stride = stride; a.v = V; a.tables = tables; a.skip = skip;
      a.state = S; a.norm_state = N; a.o_raw = o_raw; a.nq = nq;
      a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
      a.n_heads = n_heads; a.n_groups = n_groups; a.d = dk; a.dv = dv; a.from = walk_from;
      rc = launch_state_walk<WALK_LINEAR>(a, n_requests, cols, stream);
    }
    if (rc != 0 || walk_from == 1) return rc;
  }
  const int below = walk_from > 0 ? walk_from : INT_MAX;
  dim3 grid(n_requests, n_heads, (cols + LR_COLS - 1) / LR_COLS);
#define LLMRS_LR_LAUNCH(D, L)                                                                                     \
  linear_recurrence_kernel<D, L, SOME><<<grid, LR_COLS * L, 0, stream>>>(Q, K, V, decay, head_decay, v_gain, skip, S, N, \
                                                                         q_start, n_new, slot_ids, o_raw, nq, n_heads,  \
                                                                         n_groups, dk, dv, below)
  auto launch = [&](auto some) {
    constexpr bool SOME = decltype(some)::value;
    if (dk <= 32) LLMRS_LR_LAUNCH(32, 4);
    else if (dk <= 64) LLMRS_LR_LAUNCH(64, 4);
    else if (dk <= 128) LLMRS_LR_LAUNCH(128, 8);
    else LLMRS_LR_LAUNCH(256, 8);
  };
  if (walk_from > 0) launch(std::true_type());
  else launch(std::false_type());
#undef LLMRS_LR_LAUNCH
  return llmrs_launch_status("linear_recurrence");
}

// Floats of the workspace `tables` of llmrs_linear_recurrence_planes, by its walk_from: the coefficients of a portion's turns, or the
// rows of its chunks; none where no request is walked.
LLMRS_API long long llmrs_linear_recurrence_table_floats(int n_tokens, int n_requests, int n_heads, int dk, int dv, int walk_from) {
  if (walk_from <= 0) return 0;
  if (ck_takes(CK_LINEAR, dk, dv)) return ck_work_floats(CK_LINEAR, n_tokens, n_requests, walk_from, n_heads, dk, ck_columns(dv, true));
  return walk_places(n_tokens, n_requests) * n_heads * walk_table(WALK_LINEAR);
}

// Floats of workspace for llmrs_linear_recurrence: the three prepared planes and the tables.
LLMRS_API long long llmrs_linear_recurrence_work_floats(int n_tokens, int n_requests, int n_heads, int dk, int dv, int walk_from) {
  return (long long)n_tokens * n_heads * (2LL * dk + dv) + 12 +
         llmrs_linear_recurrence_table_floats(n_tokens, n_requests, n_heads, dk, dv, walk_from);
}

// q, k, v: [tokens, ...] of the activation type with their row strides, head h's channels at h * dk (h * dv);
// act 1: SiLU on all three first; rot_dims > 0: rotation of q and k with inv_freq (double [rot_dims / 2]) at `positions`;
// q is multiplied by q_scale, k by k_scale and its gain; decay [tokens, heads] or null (then head_decay [heads],
// or 1 when that is null too); gain [tokens, heads] or null (1); S [slots, heads, dk, dv]; N [slots, heads, dk] or
// null (no normaliser: nq is not written); o_raw float32 [tokens, heads * dv]; nq float32 [tokens, heads].
LLMRS_API int llmrs_linear_recurrence(const void* q, const void* k, const void* v, long long q_stride,
                                      long long k_stride, long long v_stride, int dtype, int act, float q_scale,
                                      float k_scale, const double* inv_freq, const int* positions, int rot_dims,
                                      const float* decay, const float* head_decay, const float* gain, float* S,
                                      float* N, const int* q_start, const int* n_new, const int* slot_ids,
                                      float* work, float* o_raw, float* nq, int n_tokens, int n_requests, int n_heads,
                                      int dk, int dv, int walk_from, cudaStream_t stream) {
  LLMRS_REQUIRE(n_requests >= 0 && n_tokens >= 0 && n_heads > 0 && dk > 0 && dv > 0, "linear_recurrence: bad sizes");
  LLMRS_REQUIRE(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dk, "linear_recurrence: rot_dims %d of %d", rot_dims, dk);
  LLMRS_REQUIRE(rot_dims == 0 || (inv_freq != nullptr && positions != nullptr),
                "linear_recurrence: a rotation needs frequencies and positions");
  LLMRS_REQUIRE(((uintptr_t)work & 15) == 0, "linear_recurrence: the workspace must be 16-byte aligned");
  if (n_requests == 0 || n_tokens == 0) return 0;
  // Each plane starts on a 16-byte boundary.
  const size_t nk = ((size_t)n_tokens * n_heads * dk + 3) / 4 * 4;
  float* Q = work;
  float* K = Q + nk;
  float* V = K + nk;
  float* tables = V + ((size_t)n_tokens * n_heads * dv + 3) / 4 * 4;
  const int threads = n_heads * dk >= 1024 ? 256 : 128;
  const size_t smem = (size_t)rot_dims * sizeof(float);
  auto wide = [&](int size) {      // without a rotation, every piece of sixteen bytes within a head and on a boundary
    const int piece = 16 / size;
    auto starts = [&](const void* p, long long stride) { return ((uintptr_t)p & 15) == 0 && stride % piece == 0; };
    return rot_dims == 0 && dk % piece == 0 && dv % piece == 0 && starts(q, q_stride) && starts(k, k_stride) && starts(v, v_stride);
  };
  const long long numbers = (long long)n_tokens * (2 * n_heads * dk + n_heads * dv);
#define LLMRS_LR_PREPARE(T)                                                                                            \
  do {                                                                                                                 \
    if (wide(sizeof(T)))                                                                                               \
      lr_prepare_wide_kernel<T><<<(unsigned)((numbers / (16 / (int)sizeof(T)) + 255) / 256), 256, 0, stream>>>(        \
          (const T*)q, (const T*)k, (const T*)v, q_stride, k_stride, v_stride, gain, Q, K, V, n_tokens, n_heads, dk,   \
          dv, act, q_scale, k_scale);                                                                                  \
    else                                                                                                               \
      lr_prepare_kernel<T><<<n_tokens, threads, smem, stream>>>((const T*)q, (const T*)k, (const T*)v, q_stride,       \
                                                                k_stride, v_stride, gain, inv_freq, positions,         \
                                                                rot_dims, Q, K, V, n_heads, dk, dv, act, q_scale,      \
                                                                k_scale);                                              \
  } while (0)
  if (dtype == LLMRS_F32) LLMRS_LR_PREPARE(float);
  else if (dtype == LLMRS_BF16) LLMRS_LR_PREPARE(__nv_bfloat16);
  else return llmrs_fail("linear_recurrence: unknown dtype %d", dtype);
#undef LLMRS_LR_PREPARE
  int rc = llmrs_launch_status("linear_recurrence (prepare)");
  if (rc != 0) return rc;
  return llmrs_linear_recurrence_planes(Q, K, V, decay, head_decay, nullptr, nullptr, S, N, q_start, n_new, slot_ids,
                                        tables, o_raw, nq, n_tokens, n_requests, n_heads, n_heads, dk, dv, walk_from, stream);
}

// ---------------------------------------------------------------------------------
// output: out[t, h, :] = norm(o[t, h, :] / den[t, h]) * weight * act(gate[t, h, :]); one block per token; act is the
// sigmoid, or SiLU with gate_silu; weight null: none.
// den = max(|nq|, floor) + den_eps when nq is given, else 1. per_head 1: each head is divided by its own root mean
// square; 0: all heads of a token together.
// ---------------------------------------------------------------------------------
template <typename TA>
__global__ void lr_output_kernel(const float* __restrict__ o_raw, const float* __restrict__ nq,
                                 const float* __restrict__ floor_, float den_eps, const TA* __restrict__ gate,
                                 long long gate_stride, const float* __restrict__ norm_w, TA* __restrict__ out,
                                 int n_heads, int dv, int per_head, int gate_silu, float eps) {
  extern __shared__ float sh[];      // [heads] 1 / den, then [heads] sums of squares
  __shared__ float red[33];
  float* inv_den = sh;
  float* hss = sh + n_heads;
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  const float* o = o_raw + (size_t)t * n_heads * dv;
  for (int h = warp; h < n_heads; h += n_warps) {
    float id = 1.0f;
    if (nq) id = 1.0f / (fmaxf(fabsf(nq[(size_t)t * n_heads + h]), floor_[(size_t)t * n_heads + h]) + den_eps);
    float ss = 0.f;
    for (int i = lane; i < dv; i += 32) {
      const float x = o[h * dv + i] * id;
      ss = fmaf(x, x, ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) {
      inv_den[h] = id;
      hss[h] = ss;
    }
  }
  __syncthreads();
  float all = 0.f;
  if (!per_head) {
    float s = 0.f;
    for (int h = threadIdx.x; h < n_heads; h += blockDim.x) s += hss[h];
    all = 1.0f / sqrtf(block_sum(s, red) / (float)(n_heads * dv) + eps);
  }
  for (int c = threadIdx.x; c < n_heads * dv; c += blockDim.x) {
    const int h = c / dv;
    const float inv = per_head ? 1.0f / sqrtf(hss[h] / (float)dv + eps) : all;
    const float x = to_float(gate[(size_t)t * gate_stride + c]), g = gate_silu ? rec_silu(x) : rec_sigmoid(x);
    out[(size_t)t * n_heads * dv + c] = from_float<TA>(o[c] * inv_den[h] * inv * (norm_w ? norm_w[c] : 1.0f) * g);
  }
}

LLMRS_API int llmrs_recurrence_output(const float* o_raw, const float* nq, const float* floor_, float den_eps,
                                      const void* gate, long long gate_stride, int dtype, const float* norm_w,
                                      void* out, int n_tokens, int n_heads, int dv, int per_head, int gate_silu,
                                      float eps, cudaStream_t stream) {
  LLMRS_REQUIRE(n_tokens >= 0 && n_heads > 0 && dv > 0 && n_heads <= 4096, "recurrence_output: bad sizes");
  LLMRS_REQUIRE((nq == nullptr) == (floor_ == nullptr), "recurrence_output: nq and floor come together");
  if (n_tokens == 0) return 0;
  HeadOutArgs a = {};
  a.o = o_raw; a.nq = nq; a.floor_ = floor_; a.den_eps = den_eps; a.gate = gate; a.gate_stride = gate_stride; a.w = norm_w;
  a.out = out; a.out_stride = (long long)n_heads * dv; a.n_tokens = n_tokens; a.n_heads = n_heads; a.dv = dv;
  a.eps = eps; a.out_scale = 1.0f; a.silu = gate_silu;
  if (per_head && dtype == LLMRS_F32 && head_out_takes<float>(a)) {
    launch_head_out<float>(a, stream);
    return llmrs_launch_status("recurrence_output");
  }
  if (per_head && dtype == LLMRS_BF16 && head_out_takes<__nv_bfloat16>(a)) {
    launch_head_out<__nv_bfloat16>(a, stream);
    return llmrs_launch_status("recurrence_output");
  }
  const int threads = n_heads * dv >= 2048 ? 256 : 128;
  const size_t smem = 2 * (size_t)n_heads * sizeof(float);
  if (dtype == LLMRS_F32)
    lr_output_kernel<float><<<n_tokens, threads, smem, stream>>>(o_raw, nq, floor_, den_eps, (const float*)gate,
                                                                 gate_stride, norm_w, (float*)out, n_heads, dv,
                                                                 per_head, gate_silu, eps);
  else if (dtype == LLMRS_BF16)
    lr_output_kernel<__nv_bfloat16><<<n_tokens, threads, smem, stream>>>(
        o_raw, nq, floor_, den_eps, (const __nv_bfloat16*)gate, gate_stride, norm_w, (__nv_bfloat16*)out, n_heads, dv,
        per_head, gate_silu, eps);
  else
    return llmrs_fail("recurrence_output: unknown dtype %d", dtype);
  return llmrs_launch_status("recurrence_output");
}
