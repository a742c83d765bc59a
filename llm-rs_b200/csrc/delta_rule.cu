// Generalized delta rule: a recurrent mixer whose per-head state S [key channel, value channel] is updated by
//
//   S <- diag(w) S - (a * u) (u^T S) + k v^T        (both products read the old S)
//   o  = S^T r
//
// with the unit key u = k / sqrt(sum(k^2) + key_eps), a per-channel decay w = exp(-decay_scale * sigmoid(d + d0))
// from the decay projection d, and a per-channel removal rate a = sigmoid(a_raw + a_bias). After the recurrence each
// head's o is divided by its root mean square, multiplied by a weight and by sigmoid(gate), and rounded to the
// activation type.
//
// Two kernels and a small third:
//   prepare     a warp per (token, head), all tokens at once: decay, removal rate times unit key, unit key, and r, k, v
//               widened, as six float32 rows [tokens, heads * d];
//   (requests that are walked take their rows and the walk of state_chunks.cuh instead of these two, heads of more than 64 channels
//   `turns` and the walk of state_walk.cuh; 2,048 tokens of 32 heads of 64 x 64: 816 us walked one by one, 246 in turns, 92 in
//   chunks; their rows 104 us, those of turns 56, where `prepare` takes 38)
//   recurrence  one block per (request, head, slice of 16 value columns) walks the request's tokens of the step in
//               order: a column of S depends on no other column, so the slices run side by side. Four adjacent lanes
//               share a column, each keeping a quarter of its key channels in registers; u^T S and S^T r are summed
//               over the four with two shuffles. The prepared rows come in chunks through two shared-memory buffers
//               (16-byte asynchronous copies), so the next chunk arrives while this one is walked, and are read as
//               16-byte broadcasts. The state lives in float32 per request slot, read at the start and written at the
//               end: a step of one token (decoding) and a prompt's portion are the same kernel;
//   output      divides by the head's root mean square, applies the weight and the gate (head_out.cuh; heads that it does not
//               take: a warp per token and head).
#include <limits.h>

#include "common.cuh"
#include "head_out.cuh"
#include "mma_util.cuh"
#include "state_chunks.cuh"

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

constexpr int DR_COLS = 16, DR_LANES = 4, DR_THREADS = DR_COLS * DR_LANES;
enum { DR_W = 0, DR_AU = 1, DR_U = 2, DR_K = 3, DR_R = 4, DR_V = 5, DR_ROWS = 6 };
// Planes of rows in the workspace: none where every request is walked in chunks.
static int dr_prepared(int d, int walk_from) { return walk_from == 1 && ck_takes(CK_GENERAL, d, d) ? 0 : DR_ROWS; }

// prep: float32 [6][tokens][heads * d] in the order of the enum above; of requests of fewer than `below` tokens.
template <typename TA>
__global__ void delta_prepare_kernel(const TA* __restrict__ r, const TA* __restrict__ k, const TA* __restrict__ v,
                                     const TA* __restrict__ a_raw, long long in_stride,
                                     const float* __restrict__ decay_raw, const float* __restrict__ decay_bias,
                                     const float* __restrict__ a_bias, const int* __restrict__ q_start,
                                     const int* __restrict__ n_new, float* __restrict__ prep, int n_tokens, int n_requests,
                                     int n_heads, int d, float decay_scale, float key_eps, int below) {
  const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n_tokens * n_heads) return;
  const int t = row / n_heads, h = row % n_heads;
  if (below < INT_MAX && n_new[walk_token_request(q_start, n_requests, t)] >= below) return;
  const size_t in0 = (size_t)t * in_stride + (size_t)h * d, out0 = (size_t)t * n_heads * d + (size_t)h * d;
  const size_t plane = (size_t)n_tokens * n_heads * d;
  float ss = 0.f;
  for (int i = lane; i < d; i += 32) {
    const float kv = to_float(k[in0 + i]);
    ss += kv * kv;
  }
  const float inv = 1.0f / sqrtf(warp_sum(ss) + key_eps);
  for (int i = lane; i < d; i += 32) {
    const float kv = to_float(k[in0 + i]), u = kv * inv;
    prep[DR_W * plane + out0 + i] = expf(-decay_scale * sigmoidf_(decay_raw[out0 + i] + decay_bias[h * d + i]));
    prep[DR_AU * plane + out0 + i] = sigmoidf_(to_float(a_raw[in0 + i]) + a_bias[h * d + i]) * u;
    prep[DR_U * plane + out0 + i] = u;
    prep[DR_K * plane + out0 + i] = kv;
    prep[DR_R * plane + out0 + i] = to_float(r[in0 + i]);
    prep[DR_V * plane + out0 + i] = to_float(v[in0 + i]);
  }
}

// What the walk in turns of four tokens reads (state_walk.cuh), a warp per (turn, head): r and u decayed from the turn's start
// (r with the token's own decay, u without: it meets the state before the token), k and the removal -a u decayed from the
// token to the turn's end, the whole turn's decay, v widened, and the coefficients between the turn's tokens. rows: r, u, k,
// -a u and v, each [tokens, heads * d]. vec, vec_f: the inputs' and the float32 rows' pieces of four (two with CPL 2) channels
// start on their own boundaries.
template <typename TA, int CPL>
__global__ void __launch_bounds__(128)
delta_turns_kernel(const TA* __restrict__ r, const TA* __restrict__ k, const TA* __restrict__ v, const TA* __restrict__ a_raw,
                   long long in_stride, const float* __restrict__ decay_raw, const float* __restrict__ decay_bias,
                   const float* __restrict__ a_bias, const int* __restrict__ q_start, const int* __restrict__ n_new,
                   float* __restrict__ rows, float* __restrict__ w, float* __restrict__ tables, int n_tokens, int n_requests,
                   int n_heads, int d, float decay_scale, float key_eps, bool vec, bool vec_f, int from) {
  const int place = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= n_heads) return;
  const int req = walk_request(q_start, n_requests, place), t_req = q_start[req];
  const int first = (place - walk_place(t_req, req)) * WALK_TURN, have = min(WALK_TURN, n_new[req] - first);
  if (first < 0 || have <= 0 || n_new[req] < from) return;
  const size_t t0 = (size_t)(t_req + first), width = (size_t)n_heads * d, plane = (size_t)n_tokens * width;
  float rv[4][CPL], kv[4][CPL], au[4][CPL], dec[4][CPL], bias_d[CPL], bias_a[CPL];
  walk_load<CPL>(decay_bias + (size_t)h * d, lane, d, true, false, bias_d);
  walk_load<CPL>(a_bias + (size_t)h * d, lane, d, true, false, bias_a);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const size_t in = (t0 + t) * in_stride + (size_t)h * d, at = (t0 + t) * width + (size_t)h * d;
    walk_load<CPL>(k + in, lane, d, t < have, vec, kv[t]);
    walk_load<CPL>(r + in, lane, d, t < have, vec, rv[t]);
    walk_load<CPL>(a_raw + in, lane, d, t < have, vec, au[t]);
    walk_load<CPL>(decay_raw + at, lane, d, t < have, vec_f, dec[t]);
    float value[CPL];
    walk_load<CPL>(v + in, lane, d, t < have, vec, value);
    if (t < have) walk_store<CPL>(rows + 4 * plane + at, lane, d, vec_f, value);
  }
  float u[4][CPL];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float ss = 0.f;
#pragma unroll
    for (int m = 0; m < CPL; ++m) ss = fmaf(kv[t][m], kv[t][m], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) + key_eps);
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
      u[t][m] = kv[t][m] * inv;
      au[t][m] = -sigmoidf_(au[t][m] + bias_a[m]) * u[t][m];
      dec[t][m] = t < have ? expf(-decay_scale * sigmoidf_(dec[t][m] + bias_d[m])) : 1.f;
    }
  }
  // A (u_i . a_j) at 0, B (u_i . k_j) at 6, for j < i at i (i - 1) / 2 + j; R (r_i . k_j) at 12, Q (r_i . a_j) at 22, for
  // j <= i at i (i + 1) / 2 + j: 32 sums, a lane each.
  float sums[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) sums[e] = 0.f;
#pragma unroll
  for (int m = 0; m < CPL; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float kj = kv[j][m], aj = au[j][m];      // what token j wrote, decayed up to and with token t below
      sums[12 + j * (j + 1) / 2 + j] = fmaf(rv[j][m], kj, sums[12 + j * (j + 1) / 2 + j]);
      sums[22 + j * (j + 1) / 2 + j] = fmaf(rv[j][m], aj, sums[22 + j * (j + 1) / 2 + j]);
#pragma unroll
      for (int t = j + 1; t < 4; ++t) {
        const int e = t * (t - 1) / 2 + j, f = t * (t + 1) / 2 + j;
        sums[e] = fmaf(u[t][m], aj, sums[e]);
        sums[6 + e] = fmaf(u[t][m], kj, sums[6 + e]);
        kj *= dec[t][m];
        aj *= dec[t][m];
        sums[12 + f] = fmaf(rv[t][m], kj, sums[12 + f]);
        sums[22 + f] = fmaf(rv[t][m], aj, sums[22 + f]);
      }
    }
  float up[CPL], down[CPL], row[CPL];
#pragma unroll
  for (int m = 0; m < CPL; ++m) up[m] = down[m] = 1.f;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int e = 3 - t;
    if (t < have) {
      const size_t at = (t0 + t) * width + (size_t)h * d;
#pragma unroll
      for (int m = 0; m < CPL; ++m) row[m] = u[t][m] * up[m];
      walk_store<CPL>(rows + plane + at, lane, d, vec_f, row);
#pragma unroll
      for (int m = 0; m < CPL; ++m) row[m] = rv[t][m] * (up[m] * dec[t][m]);
      walk_store<CPL>(rows + at, lane, d, vec_f, row);
    }
    if (e < have) {
      const size_t at = (t0 + e) * width + (size_t)h * d;
#pragma unroll
      for (int m = 0; m < CPL; ++m) row[m] = kv[e][m] * down[m];
      walk_store<CPL>(rows + 2 * plane + at, lane, d, vec_f, row);
#pragma unroll
      for (int m = 0; m < CPL; ++m) row[m] = au[e][m] * down[m];
      walk_store<CPL>(rows + 3 * plane + at, lane, d, vec_f, row);
    }
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
      up[m] *= dec[t][m];
      down[m] *= dec[e][m];
    }
  }
  walk_store<CPL>(w + ((size_t)place * n_heads + h) * d, lane, d, vec_f, up);
  float* to = tables + ((size_t)place * n_heads + h) * 48;
  const float sum = walk_sum_all<32>(sums, lane);
  if (lane < 12) {
    to[lane < 6 ? WALK_GA + lane : WALK_GB + lane - 6] = sum;
  } else {
    const int f = lane < 22 ? lane - 12 : lane - 22, i = f < 1 ? 0 : (f < 3 ? 1 : (f < 6 ? 2 : 3));
    to[(lane < 22 ? WALK_GR : WALK_GQ) + 4 * i + f - i * (i + 1) / 2] = sum;
  }
  if (lane < 12) {      // above the diagonals
    const int e = lane % 6;
    to[(lane < 6 ? WALK_GR : WALK_GQ) + (e < 3 ? 1 + e : (e < 5 ? 3 + e : 11))] = 0.f;
  }
}

// The same for chunks of sixteen tokens (state_chunks.cuh), heads of at most 64 channels: a block per (place, head). Half a warp
// walks a token j through the tokens after it, the decays multiplied on as they go, and then token 15 - j, so that every one has
// seventeen steps; then a warp makes the rows of sixteen channels, which are sixteen value columns too.
template <typename TA>
struct DeltaRowsArgs {
  const TA *r, *k, *v, *a_raw;
  long long in_stride;
  const float *decay_raw, *decay_bias, *a_bias;
  const int *q_start, *n_new;
  float *tiles, *u_out, *g_out, *v_out;
  int n_requests, n_heads, d;
  float decay_scale, key_eps;
  int from;
};
struct DeltaRowsShared {
  alignas(16) __nv_bfloat16 E[CK_MATRIX], R[CK_MATRIX], Q[CK_MATRIX], T[CK_MATRIX];
  float sums[4][CK][CK + 1];      // u_i . k_j, u_i . a_j, r_i . k_j, r_i . a_j
};
// True where CAREFUL would make something else of it.
template <typename TA, bool CAREFUL>
__device__ __forceinline__ bool delta_rows(const DeltaRowsArgs<TA>& p, float* tile, DeltaRowsShared& sh) {
  constexpr int GS = CK + 1, DMAX = 64, RS = DMAX + 4, ROW = DMAX + 8;
  const TA *r = p.r, *k = p.k, *v = p.v, *a_raw = p.a_raw;
  const long long in_stride = p.in_stride;
  const float *decay_raw = p.decay_raw, *decay_bias = p.decay_bias, *a_bias = p.a_bias;
  const int *q_start = p.q_start, *n_new = p.n_new;
  const int n_requests = p.n_requests, n_heads = p.n_heads, d = p.d, from = p.from;
  const float decay_scale = p.decay_scale, key_eps = p.key_eps;
  float* tile_out = p.tiles + ((size_t)blockIdx.x * n_heads + blockIdx.y) * ck_tile(CK_GENERAL, DMAX);
  auto ks = reinterpret_cast<float (*)[RS]>(tile + ck_rows(2, DMAX));      // (two planes of the tile at a time: four blocks an SM)
  auto rs = ks + CK, us = rs + CK, as = us + CK, ws = as + CK;
  auto &E = sh.E, &R = sh.R, &Q = sh.Q, &T = sh.T;
  auto& sums = sh.sums;
  CkLook look;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int place = blockIdx.x;
  int t_req, n_req;
  const int place0 = ck_request(q_start, n_new, n_requests, from, place, t_req, n_req);
  const int first = (place - place0) * CK, have = min(CK, n_req - first);
  if (first < 0 || have <= 0 || n_req < from) return false;
  const size_t t0 = (size_t)(t_req + first), width = (size_t)n_heads * d;
  {
    float kv[CK / 4][2], rv[CK / 4][2], av[CK / 4][2], dec[CK / 4][2], bias_a[2], bias_d[2];      // a warp a token, all on their way together
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int c = lane + 32 * m;
      const size_t ch = (size_t)h * d + c;
      bias_a[m] = c < d ? a_bias[ch] : 0.f;
      bias_d[m] = c < d ? decay_bias[ch] : 0.f;
#pragma unroll
      for (int x = 0; x < CK / 4; ++x) {
        const int t = 4 * x + warp;
        const size_t at = (t0 + t) * in_stride + ch;
        kv[x][m] = rv[x][m] = av[x][m] = dec[x][m] = 0.f;
        if (t < have && c < d) {
          kv[x][m] = to_float(k[at]);
          rv[x][m] = to_float(r[at]);
          av[x][m] = to_float(a_raw[at]);
          dec[x][m] = decay_raw[(t0 + t) * width + ch];
        }
      }
    }
#pragma unroll
    for (int x = 0; x < CK / 4; ++x) {
      const int t = 4 * x + warp;
      const float inv = 1.0f / sqrtf(warp_sum(fmaf(kv[x][0], kv[x][0], kv[x][1] * kv[x][1])) + key_eps);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int c = lane + 32 * m;
        const bool there = t < have && c < d;
        const float u = there ? kv[x][m] * inv : 0.f;
        ks[t][c] = kv[x][m];
        us[t][c] = u;
        rs[t][c] = rv[x][m];
        as[t][c] = there ? -sigmoidf_(av[x][m] + bias_a[m]) * u : 0.f;
        ws[t][c] = there ? expf(-decay_scale * sigmoidf_(dec[x][m] + bias_d[m])) : 1.f;
      }
    }
  }
  // The values that this warp needs below are on their way.
  const int c0 = 16 * warp;
  float value[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int t = ck_token(lane, e), c = c0 + ck_channel(lane, e);
    value[e] = t < have && c < d ? to_float(v[(t0 + t) * in_stride + (size_t)h * d + c]) : 0.f;
  }
  __syncthreads();
  {
    const int pair = tid >> 4, at = (tid & 15) * 4;
    auto four = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
    auto dot = [](const float4& x, const float4& y) { return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, x.w * y.w))); };
    auto times = [](float4& x, const float4& w) { x.x *= w.x; x.y *= w.y; x.z *= w.z; x.w *= w.w; };
    float4 kj = four(&ks[pair][at]), aj = four(&as[pair][at]);
    for (int step = 0; step <= CK; ++step) {      // token `pair` through the tokens from it on, then token 15 - pair
      const bool second = step >= CK - pair;
      const int j = second ? CK - 1 - pair : pair, i = second ? step - 1 : pair + step;
      if (step == CK - pair) {
        kj = four(&ks[j][at]);
        aj = four(&as[j][at]);
      }
      const float4 u = four(&us[i][at]), x = four(&rs[i][at]), w = four(&ws[i][at]);
      const float uk = dot(u, kj), ua = dot(u, aj);      // with the decays up to the token before i
      if (i > j) {
        times(kj, w);
        times(aj, w);
      }
      const float rk = dot(x, kj), ra = dot(x, aj);      // with i's own too
      // Four sums over sixteen lanes: lane bits 3 and 2 say whose.
      const bool b3 = tid & 8, b2 = tid & 4;
      const float x0 = (b3 ? rk : uk) + __shfl_xor_sync(0xffffffffu, b3 ? uk : rk, 8);
      const float x1 = (b3 ? ra : ua) + __shfl_xor_sync(0xffffffffu, b3 ? ua : ra, 8);
      float s = (b2 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, b2 ? x0 : x1, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if ((tid & 3) == 0) sums[tid >> 2 & 3][i][j] = s;
    }
  }
  __syncthreads();
  // The rows with their decays: u and r from the chunk's start, k and a to its end. Beside that the system.
  if (tid < DMAX) {
    float up = 1.f, down = 1.f;
#pragma unroll
    for (int t = CK - 1; t >= 0; --t) {
      ks[t][tid] *= down;
      as[t][tid] *= down;
      down *= ws[t][tid];
    }
#pragma unroll
    for (int t = 0; t < CK; ++t) {
      us[t][tid] *= up;
      up *= ws[t][tid];
      rs[t][tid] *= up;
    }
    tile_out[ck_rows(CK_GENERAL, DMAX) + tid] = up;
  } else if (warp == 3) {
    if (lane < CK) ck_solve<CAREFUL>(&sums[1][0][0], GS, -1.f, lane, 1.f, T);
  } else {
    for (int e = lane; e < CK * CK; e += 32) {
      const int i = e / CK, j = e % CK;
      ck_set<CAREFUL>(E, i, j, j < i ? sums[0][i][j] : 0.f);
      ck_set<CAREFUL>(R, i, j, j <= i ? sums[2][i][j] : 0.f);
      ck_set<CAREFUL>(Q, i, j, j <= i ? sums[3][i][j] : 0.f);
    }
  }
  __syncthreads();
  {
    uint32_t a[3][4];
    float x[8], f[8];
    auto rows_of = [&](const float (*m)[RS], float (&y)[8]) {
#pragma unroll
      for (int e = 0; e < 8; ++e) y[e] = m[ck_token(lane, e)][c0 + ck_channel(lane, e)];
    };
    rows_of(us, x);
    rows_of(rs, f);
    ck_system_rows<CAREFUL>(tile, 1, ROW, c0, lane, T, Q, x, f, look);
    ck_operand_of<CAREFUL>(f, a, look);
    ck_put(tile, 0, ROW, c0, lane, a);
    ck_tile_written();
    __syncthreads();
    if (tid == 0) {
      ck_tile_leaves(tile_out + CK_F * ck_rows(1, DMAX), tile, ck_rows(1, DMAX));
      ck_tile_leaves(tile_out + CK_W * ck_rows(1, DMAX), tile + ck_rows(1, DMAX), ck_rows(1, DMAX));
      ck_tile_left();
    }
  }
  {
    float e_v[8], y[8], o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) e_v[e] = y[e] = o[e] = 0.f;
    ck_apply<CAREFUL>(R, value, lane, o, look);
    ck_apply<CAREFUL>(E, value, lane, e_v, look);
    ck_apply<CAREFUL>(T, e_v, lane, y, look);
    ck_apply<CAREFUL>(Q, y, lane, o, look);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int t = ck_token(lane, e), c = c0 + ck_channel(lane, e);
      if (t < have && c < d) {
        const size_t to = (t0 + t) * width + (size_t)h * d + c;
        p.v_out[to] = value[e];
        p.u_out[to] = y[e];
        p.g_out[to] = o[e];
      }
    }
  }
  __syncthreads();      // F and W have left
  if (tid == 0) tile[DMAX / 2] = __int_as_float(CAREFUL);      // (B's flag: the place of B is that of F now)
#pragma unroll
  for (int plane = 0; plane < 2; ++plane) {
    uint32_t a[3][4];
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = (plane ? ks : as)[ck_token(lane, e)][c0 + ck_channel(lane, e)];
    ck_operand_of<CAREFUL>(x, a, look);
    ck_put(tile, plane, ROW, c0, lane, a);
  }
  ck_tile_written();
  __syncthreads();
  if (tid == 0) {
    ck_tile_leaves(tile_out + CK_B * ck_rows(1, DMAX), tile, ck_rows(1, DMAX));
    ck_tile_leaves(tile_out + CK_C * ck_rows(1, DMAX), tile + ck_rows(1, DMAX), ck_rows(1, DMAX));
    ck_tile_left();
  }
  return !CAREFUL && look.found();
}
template <typename TA>
__device__ __noinline__ void delta_rows_carefully(const DeltaRowsArgs<TA>& p, float* tile, DeltaRowsShared& sh) {
  ck_tile_again();
  delta_rows<TA, true>(p, tile, sh);
}
template <typename TA>
__global__ void __launch_bounds__(128, 4) delta_rows_kernel(const __grid_constant__ DeltaRowsArgs<TA> p) {
  extern __shared__ __align__(128) float dr_raw[];
  __shared__ DeltaRowsShared sh;
  if (__syncthreads_or(delta_rows<TA, false>(p, dr_raw, sh))) delta_rows_carefully<TA>(p, dr_raw, sh);
}

// SOME: only requests of fewer than `below` tokens, the others are walked in turns. (A template: with the test in it the kernel
// that takes all requests was compiled to 135 registers instead of 157 and took 115 us instead of 108.)
template <int DMAX, bool SOME>
__global__ void __launch_bounds__(DR_THREADS)
delta_rule_kernel(const float* __restrict__ prep, float* __restrict__ state, const int* __restrict__ q_start,
                  const int* __restrict__ n_new, const int* __restrict__ slot_ids, float* __restrict__ o_raw,
                  int n_tokens, int n_heads, int d, int below) {
  constexpr int CHUNK = DMAX >= 256 ? 4 : (DMAX >= 128 ? 8 : 16);
  constexpr int IPL = DMAX / DR_LANES;             // key channels per lane
  __shared__ __align__(16) float s_in[2][5][CHUNK][DMAX];      // W, AU, U, K, R of a chunk's tokens; channels >= d stay 0
  __shared__ __align__(16) float s_v[2][CHUNK][DR_COLS];
  const int req = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * DR_COLS;
  const int tid = threadIdx.x;
  const int col = col0 + tid / DR_LANES, part = tid % DR_LANES, i0 = part * IPL;
  const bool live = col < d;
  const int t0 = q_start[req], n = n_new[req];
  if (SOME && n >= below) return;
  const int ch0 = head * d, width = n_heads * d;
  const size_t plane = (size_t)n_tokens * width;
  float* S_g = state + ((size_t)slot_ids[req] * n_heads + head) * d * d;
  float S[IPL];
#pragma unroll
  for (int i = 0; i < IPL; ++i) S[i] = (live && i0 + i < d) ? S_g[(size_t)(i0 + i) * d + col] : 0.f;
  for (int e = tid; e < 2 * 5 * CHUNK * DMAX; e += DR_THREADS) (&s_in[0][0][0][0])[e] = 0.f;
  for (int e = tid; e < 2 * CHUNK * DR_COLS; e += DR_THREADS) (&s_v[0][0][0])[e] = 0.f;
  __syncthreads();
  // 16-byte copies when every row starts on a 16-byte boundary, else element by element.
  const bool wide = d % 4 == 0;
  const int ncols = min(DR_COLS, d - col0);
  auto load_chunk = [&](int buf, int c0) {
    const int cn = min(CHUNK, n - c0);
    if (wide) {
      const int per_row = d / 4;
      for (int e = tid; e < 5 * cn * per_row; e += DR_THREADS) {
        const int a = e / (cn * per_row), rem = e % (cn * per_row), tt = rem / per_row, piece = rem % per_row;
        cp_async_16(&s_in[buf][a][tt][piece * 4], prep + a * plane + (size_t)(t0 + c0 + tt) * width + ch0 + piece * 4, 16);
      }
    } else {
      for (int e = tid; e < 5 * cn * d; e += DR_THREADS) {
        const int a = e / (cn * d), rem = e % (cn * d), tt = rem / d, i = rem % d;
        s_in[buf][a][tt][i] = prep[a * plane + (size_t)(t0 + c0 + tt) * width + ch0 + i];
      }
    }
    for (int e = tid; e < cn * ncols; e += DR_THREADS) {
      const int tt = e / ncols, c = e % ncols;
      s_v[buf][tt][c] = prep[DR_V * plane + (size_t)(t0 + c0 + tt) * width + ch0 + col0 + c];
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
    for (int tt = 0; tt < cn; ++tt) {      // unrolled: the next tokens' rows are fetched under this token's shuffles
      const float vj = s_v[buf][tt][tid / DR_LANES];
      float us[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < IPL; i += 4) {
        const float4 u4 = *reinterpret_cast<const float4*>(&s_in[buf][DR_U][tt][i0 + i]);
        us[0] = fmaf(u4.x, S[i], us[0]);
        us[1] = fmaf(u4.y, S[i + 1], us[1]);
        us[2] = fmaf(u4.z, S[i + 2], us[2]);
        us[3] = fmaf(u4.w, S[i + 3], us[3]);
      }
      float uS = (us[0] + us[1]) + (us[2] + us[3]);
      uS += __shfl_xor_sync(0xffffffffu, uS, 1);
      uS += __shfl_xor_sync(0xffffffffu, uS, 2);
      float os[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < IPL; i += 4) {
        const float4 w4 = *reinterpret_cast<const float4*>(&s_in[buf][DR_W][tt][i0 + i]);
        const float4 a4 = *reinterpret_cast<const float4*>(&s_in[buf][DR_AU][tt][i0 + i]);
        const float4 k4 = *reinterpret_cast<const float4*>(&s_in[buf][DR_K][tt][i0 + i]);
        const float4 r4 = *reinterpret_cast<const float4*>(&s_in[buf][DR_R][tt][i0 + i]);
        S[i] = fmaf(k4.x, vj, fmaf(-a4.x, uS, w4.x * S[i]));
        S[i + 1] = fmaf(k4.y, vj, fmaf(-a4.y, uS, w4.y * S[i + 1]));
        S[i + 2] = fmaf(k4.z, vj, fmaf(-a4.z, uS, w4.z * S[i + 2]));
        S[i + 3] = fmaf(k4.w, vj, fmaf(-a4.w, uS, w4.w * S[i + 3]));
        os[0] = fmaf(S[i], r4.x, os[0]);
        os[1] = fmaf(S[i + 1], r4.y, os[1]);
        os[2] = fmaf(S[i + 2], r4.z, os[2]);
        os[3] = fmaf(S[i + 3], r4.w, os[3]);
      }
      float o = (os[0] + os[1]) + (os[2] + os[3]);
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      if (part == 0 && live) o_raw[(size_t)(t0 + c0 + tt) * width + ch0 + col] = o;
    }
    __syncthreads();
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < IPL; ++i)
      if (i0 + i < d) S_g[(size_t)(i0 + i) * d + col] = S[i];
  }
}

// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * weight[h, :] * sigmoid(gate[t, h, :]); a warp per (t, h).
template <typename TA>
__global__ void delta_out_kernel(const float* __restrict__ o_raw, const TA* __restrict__ gate, long long gate_stride,
                                 const float* __restrict__ norm_w, TA* __restrict__ out, int n_rows, int n_heads,
                                 int d, float eps) {
  const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int t = row / n_heads, h = row % n_heads;
  const float* o = o_raw + (size_t)t * n_heads * d + (size_t)h * d;
  float ss = 0.f;
  for (int i = lane; i < d; i += 32) ss += o[i] * o[i];
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)d + eps);
  for (int i = lane; i < d; i += 32) {
    const float g = sigmoidf_(to_float(gate[(size_t)t * gate_stride + h * d + i]));
    out[(size_t)t * n_heads * d + (size_t)h * d + i] = from_float<TA>(o[i] * inv * norm_w[h * d + i] * g);
  }
}

template <typename TA>
static int launch_delta_out(const float* o_raw, const void* gate, long long gate_stride, const float* norm_w, void* out,
                            int n_tokens, int n_heads, int d, float eps, cudaStream_t stream) {
  HeadOutArgs a = {};
  a.o = o_raw; a.gate = gate; a.gate_stride = gate_stride; a.w = norm_w; a.out = out; a.out_stride = (long long)n_heads * d;
  a.n_tokens = n_tokens; a.n_heads = n_heads; a.dv = d; a.eps = eps; a.out_scale = 1.0f;
  const int rows = n_tokens * n_heads;
  if (head_out_takes<TA>(a)) launch_head_out<TA>(a, stream);
  else
    delta_out_kernel<TA><<<(rows + 3) / 4, 128, 0, stream>>>(o_raw, (const TA*)gate, gate_stride, norm_w, (TA*)out, rows,
                                                             n_heads, d, eps);
  return llmrs_launch_status("delta_rule (norm and gate)");
}

template <typename TA>
static int launch_delta(int dmax, dim3 grid, cudaStream_t stream, const void* r, const void* k, const void* v,
                        const void* gate, const void* a_raw, long long in_stride, const float* decay_raw,
                        const float* decay_bias, const float* a_bias, const float* norm_w, float* state,
                        const int* q_start, const int* n_new, const int* slot_ids, float* work, void* out,
                        int n_tokens, int n_requests, int n_heads, int d, float decay_scale, float key_eps,
                        float norm_eps, int walk_from) {
  const int rows = n_tokens * n_heads;
  float* prep = work;
  const int prepared = dr_prepared(d, walk_from);      // planes ahead of the read-outs
  float* o_raw = work + (size_t)prepared * rows * d;
  if (walk_from > 0) {
    auto up4 = [](size_t v) { return (v + 3) & ~(size_t)3; };
    int rc;
    if (ck_takes(CK_GENERAL, d, d)) {
      const size_t plane = (size_t)rows * d;
      float *u = work + up4((size_t)(prepared + 1) * rows * d), *g = u + plane, *v_rows = g + plane, *tiles = v_rows + plane;
      constexpr size_t smem_rows = 4 * (ck_rows(2, 64) + 5 * CK * 68);
      cudaError_t e = cudaFuncSetAttribute(delta_rows_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_rows);
      if (e != cudaSuccess) return llmrs_fail("delta_rule: shared memory %zu: %s", smem_rows, cudaGetErrorString(e));
      delta_rows_kernel<TA><<<dim3((unsigned)ck_places(n_tokens, n_requests, walk_from), n_heads), 128, smem_rows, stream>>>(
          {(const TA*)r, (const TA*)k, (const TA*)v, (const TA*)a_raw, in_stride, decay_raw, decay_bias, a_bias, q_start, n_new, tiles,
           u, g, v_rows, n_requests, n_heads, d, decay_scale, key_eps, walk_from});
      rc = llmrs_launch_status("delta_rule (chunks)");
      if (rc != 0) return rc;
      ChunkArgs a = {};
      a.tiles = tiles; a.u = u; a.g = g; a.v = v_rows; a.state = state; a.o_raw = o_raw;
      a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
      a.n_heads = n_heads; a.d = a.dv = a.columns = d; a.from = walk_from;
      rc = launch_state_chunks<CK_GENERAL>(a, n_requests, stream);
    } else {
      const size_t places = (size_t)walk_places(n_tokens, n_requests), plane = (size_t)rows * d;
      float* w = work + up4((size_t)(DR_ROWS + 1) * rows * d);
      float* tables = w + up4(places * n_heads * d);
      const dim3 grid_t((unsigned)places, (n_heads + 3) / 4);
      const int piece = d <= 64 ? 2 : 4;
      auto starts = [&](const void* p, size_t size) { return ((uintptr_t)p & (piece * size - 1)) == 0; };
      const bool vec_f = d % piece == 0 && starts(decay_raw, 4);
      const bool vec = d % piece == 0 && in_stride % piece == 0 && starts(r, sizeof(TA)) && starts(k, sizeof(TA)) &&
                       starts(v, sizeof(TA)) && starts(a_raw, sizeof(TA));
#define LLMRS_DR_TURNS(CPL)                                                                                               \
    delta_turns_kernel<TA, CPL><<<grid_t, 128, 0, stream>>>((const TA*)r, (const TA*)k, (const TA*)v, (const TA*)a_raw, in_stride, \
                                                            decay_raw, decay_bias, a_bias, q_start, n_new, prep, w, tables, \
                                                            n_tokens, n_requests, n_heads, d, decay_scale, key_eps, vec, vec_f, \
                                                            walk_from)
      if (d <= 64) LLMRS_DR_TURNS(2);
      else if (d <= 128) LLMRS_DR_TURNS(4);
      else LLMRS_DR_TURNS(8);
#undef LLMRS_DR_TURNS
      rc = llmrs_launch_status("delta_rule (turns)");
      if (rc != 0) return rc;
      WalkArgs a = {};
      a.q = prep; a.k = prep + plane; a.kb = prep + 2 * plane; a.ab = prep + 3 * plane; a.v = prep + 4 * plane; a.w = w;
      a.q_stride = a.k_stride = a.b_stride = (long long)n_heads * d;
      a.tables = tables; a.state = state; a.o_raw = o_raw;
      a.q_start = q_start; a.n_new = n_new; a.slot_ids = slot_ids;
      a.n_heads = a.n_groups = n_heads; a.d = a.dv = d; a.from = walk_from;
      rc = launch_state_walk<WALK_GENERAL>(a, n_requests, d, stream);
    }
    if (rc != 0) return rc;
    if (walk_from == 1) return launch_delta_out<TA>(o_raw, gate, in_stride, norm_w, out, n_tokens, n_heads, d, norm_eps, stream);
  }
  const int below = walk_from > 0 ? walk_from : INT_MAX;
  delta_prepare_kernel<TA><<<(rows + 3) / 4, 128, 0, stream>>>((const TA*)r, (const TA*)k, (const TA*)v,
                                                               (const TA*)a_raw, in_stride, decay_raw, decay_bias,
                                                               a_bias, q_start, n_new, prep, n_tokens, n_requests, n_heads, d,
                                                               decay_scale, key_eps, below);
  int rc = llmrs_launch_status("delta_rule (prepare)");
  if (rc != 0) return rc;
#define LLMRS_DR_WALK(D)                                                                                                     \
  do {                                                                                                                      \
    if (walk_from > 0)                                                                                                      \
      delta_rule_kernel<D, true><<<grid, DR_THREADS, 0, stream>>>(prep, state, q_start, n_new, slot_ids, o_raw, n_tokens,   \
                                                                  n_heads, d, below);                                       \
    else                                                                                                                    \
      delta_rule_kernel<D, false><<<grid, DR_THREADS, 0, stream>>>(prep, state, q_start, n_new, slot_ids, o_raw, n_tokens,  \
                                                                   n_heads, d, below);                                      \
  } while (0)
  if (dmax == 32) LLMRS_DR_WALK(32);
  else if (dmax == 64) LLMRS_DR_WALK(64);
  else if (dmax == 128) LLMRS_DR_WALK(128);
  else LLMRS_DR_WALK(256);
#undef LLMRS_DR_WALK
  rc = llmrs_launch_status("delta_rule");
  if (rc != 0) return rc;
  return launch_delta_out<TA>(o_raw, gate, in_stride, norm_w, out, n_tokens, n_heads, d, norm_eps, stream);
}

// Float32 workspace of the kernels, in floats: the prepared rows, the read-outs and, where requests are walked (walk_from as below), what
// their walk reads.
LLMRS_API long long llmrs_delta_rule_work_floats(int n_tokens, int n_requests, int n_heads, int d, int walk_from) {
  const long long plane = (long long)n_tokens * n_heads * d, base = (dr_prepared(d, walk_from) + 1) * plane + 16;
  if (walk_from <= 0) return base;
  if (ck_takes(CK_GENERAL, d, d)) return base + ck_work_floats(CK_GENERAL, n_tokens, n_requests, walk_from, n_heads, d, d) + plane;
  return base + walk_places(n_tokens, n_requests) * n_heads * (d + walk_table(WALK_GENERAL));
}

// r, k, v, gate, a_raw: [tokens, ...] of the activation type, rows `in_stride` elements apart, each pointing at its
// own first column (head h's channels at h * d); decay_raw: float32 [tokens, heads * d]; work: float32 workspace of
// llmrs_delta_rule_work_floats, 16-byte aligned; out: [tokens, heads * d]. walk_from: requests of at least so many tokens are
// walked in turns, the others token by token; 0: all of them are.
LLMRS_API int llmrs_delta_rule(const void* r, const void* k, const void* v, const void* gate, const void* a_raw,
                               long long in_stride, int dtype, const float* decay_raw, const float* decay_bias,
                               const float* a_bias, const float* norm_w, float* state, const int* q_start,
                               const int* n_new, const int* slot_ids, float* work, void* out, int n_tokens,
                               int n_requests, int n_heads, int d, float decay_scale, float key_eps, float norm_eps,
                               int walk_from, cudaStream_t stream) {
  LLMRS_REQUIRE(n_requests >= 0 && n_tokens >= 0 && n_heads > 0 && d > 0, "delta_rule: bad sizes");
  LLMRS_REQUIRE(d <= 256, "delta_rule: heads of at most 256 channels, got %d", d);
  LLMRS_REQUIRE(n_heads <= 65535, "delta_rule: too many heads");
  LLMRS_REQUIRE(((uintptr_t)work & 15) == 0, "delta_rule: the workspace must be 16-byte aligned");
  if (n_requests == 0 || n_tokens == 0) return 0;
  const int dmax = d <= 32 ? 32 : (d <= 64 ? 64 : (d <= 128 ? 128 : 256));
  dim3 grid(n_requests, n_heads, (d + DR_COLS - 1) / DR_COLS);
  if (dtype == LLMRS_F32)
    return launch_delta<float>(dmax, grid, stream, r, k, v, gate, a_raw, in_stride, decay_raw, decay_bias, a_bias,
                               norm_w, state, q_start, n_new, slot_ids, work, out, n_tokens, n_requests, n_heads, d,
                               decay_scale, key_eps, norm_eps, walk_from);
  if (dtype == LLMRS_BF16)
    return launch_delta<__nv_bfloat16>(dmax, grid, stream, r, k, v, gate, a_raw, in_stride, decay_raw, decay_bias,
                                       a_bias, norm_w, state, q_start, n_new, slot_ids, work, out, n_tokens, n_requests,
                                       n_heads, d, decay_scale, key_eps, norm_eps, walk_from);
  return llmrs_fail("delta_rule: unknown dtype %d", dtype);
}
