// The walk of state_walk.cuh in chunks of sixteen tokens, its products on the tensor cores (mma.sync). What a chunk's tokens do to
// one another does not depend on the state and is worked out for all chunks at once, ahead of the walk, as rows of key
// channels and of value columns; with S the state before a chunk, the walk itself is
//
//   Y = U + W S,   O = F S + G,   S <- D S + B^T Y (+ C^T V)
//
// where, i and j the chunk's tokens, P_i the decay up to and with i, Z_j after j, Q, K, A, R, E the coefficients of state_walk.cuh
// (Q, K, A: read-outs and systems over what tokens write, R, E: the same over the values of the generalized rule):
//
//   linear         U = gain V            no W                    F = P q               G = Q U (+ skip V)    B = Z k
//   gated          U = T V               W = -T P k              F = P q + Q W         the same              B = Z k
//                  T = (I + diag(beta) K)^-1 diag(beta); with a decay per key channel P and Z lie in the rows
//   generalized    U = T E V             W = T u                 F = r + Q W           G = R V + Q U         B = a, C = k
//                  T = (I - A)^-1, the rows decayed from the chunk's start (u, r) or to its end (a, k)
//
// Rows are sums over tokens up to their own and nothing else, so a token that is not finite leaves earlier read-outs alone. An infinite
// value or state is one in its own column, as it is token by token, and a finite one stays finite up to the end of the range (CK_LARGE).
//
// Nothing is held in fewer than 32 bits. A float32 operand x goes into the tensor cores as three bfloat16 numbers, x = x0 + x1 + x2
// with x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1): 24 bits, and a product of two such operands is the six products
// x0 y0, x0 y1, x1 y0, x1 y1, x0 y2, x2 y0 (those left out are below 2^-24 of it). The five small ones are summed apart from
// x0 y0; the state is updated by a float32 multiply-add, not inside the tensor cores, whose sums are cut off instead of rounded.
//
// A block takes 16 value columns of a head. Four warps hold the state transposed, [column][channel], in accumulators (a quarter of
// the channels each), where two neighbouring tiles of an accumulator are an operand of the next product as they stand: W S, one
// exchange of the four warps' sums, the update. Four more make the read-outs, off the chain of the walk, from the state's pieces that
// the first four leave in shared memory, and four copy the chunks to come. The rows arrive split into pieces and laid out
// as they stand in shared memory: split in here, every block of a head would do it again.
//
// Precision, float32 models of 300 tokens, states against 64 bits (in turns on the CUDA cores -> here): gated 9.7e-7 -> 5.5e-7, channel
// decays 9.2e-7 -> 5.0e-7, generalized 8.7e-7 -> 4.8e-7, linear with one decay a head 7.3e-7 -> 2.5e-7 (its decays as stored).
//
// What bounds it: one warp a scheduler walks, and a chunk is the chain state's pieces -> W S -> exchange -> Y's pieces -> update (900 ns
// of which 48 products issue for 200); the read-outs' products share the tensor cores with it, and the copies come just in time: tiles
// that do not start on lines of 128 bytes cost the gated walk 29 %. 2,048 tokens, the walk
// alone, in turns of four on the CUDA cores -> here: gated, 16 heads of 128 x 128 267 -> 117 us, generalized, 32 heads of 64 x 64
// 251 -> 92, linear with a normaliser, 1,311 tokens 184 -> 81. (Sixteen tokens with the rows split in here by the copying warps, the
// system and the read-outs on the walking warps: 193 us. Read-outs of the chunk that is walked, not of the one before: linear 90
// against 84.)
#pragma once
#include <algorithm>
#include <utility>

#include "state_walk.cuh"

constexpr int CK = 16, CK_COLS = 16, CK_WARPS = 4, CK_THREADS = 3 * 32 * CK_WARPS, CK_STAGES = 4;
// Planes of rows: F, B; W where there is one; C.
enum { CK_F = 0, CK_B = 1, CK_W = 2, CK_C = 3 };
enum { CK_LINEAR = 2, CK_SYSTEM = 3, CK_GENERAL = 4 };      // the kinds, by their planes

// A chunk's rows of one head, in floats: the planes' pieces [planes][3][16][dmax + 8] bfloat16 (eight numbers beyond a row keep
// neighbouring rows' reads in different banks), then the chunk's decay D [dmax]. (Whole lines of 128 bytes.)
__host__ __device__ constexpr int ck_rows(int planes, int dmax) { return planes * 3 * CK * (dmax + 8) / 2; }
__host__ __device__ constexpr int ck_tile(int planes, int dmax) { return ck_rows(planes, dmax) + dmax; }
// Beyond the first row of B: a word that is not zero where a number that the chunk writes is large or not finite (CK_LARGE).
__host__ __device__ constexpr int ck_flag(int dmax) { return CK_B * ck_rows(1, dmax) + dmax / 2; }
__host__ __device__ constexpr int ck_dmax(int d) { return d <= 64 ? 64 : 128; }
// Places of chunks among all chunks: a walked request's start in sixteens and its rank among the walked ones. Where all requests are
// walked (from 1) that is its number, with the requests of no tokens; otherwise those with `from` tokens and more are counted, so that
// a step's short requests take no places.
__host__ __device__ inline int ck_place(int q_start, int rank) { return q_start / CK + rank; }
inline long long ck_places(int n_tokens, int n_requests, int from) {
  return (long long)n_tokens / CK + (from <= 1 ? n_requests : std::min(n_requests, n_tokens / from)) + 1;
}
// All lanes of a warp call these two. A request's rank:
__device__ __forceinline__ int ck_rank(const int* __restrict__ n_new, int req, int from) {
  if (from <= 1) return req;
  int rank = 0;
  for (int base = 0; base < req; base += 32) {
    const int r = base + (threadIdx.x & 31);
    rank += __popc(__ballot_sync(0xffffffffu, r < req && n_new[r] >= from));
  }
  return rank;
}
// The first place, start and tokens of the request whose chunks place p lies among (the last walked one that starts at or before it).
__device__ __forceinline__ int ck_request(const int* __restrict__ q_start, const int* __restrict__ n_new, int n_requests, int from, int p,
                                          int& start, int& tokens) {
  int place = 0, rank = 0;
  start = tokens = 0;
  for (int base = 0; base < n_requests; base += 32) {
    const int lane = threadIdx.x & 31, r = base + lane;
    const int q = r < n_requests ? q_start[r] : 0, n = r < n_requests ? n_new[r] : 0;
    const unsigned walked = __ballot_sync(0xffffffffu, r < n_requests && (from <= 1 || n >= from));
    const int at = ck_place(q, rank + __popc(walked & ((1u << lane) - 1u)));
    const unsigned hit = __ballot_sync(0xffffffffu, (walked >> lane & 1u) && at <= p);
    if (hit == 0 && walked != 0) break;
    if (hit != 0) {
      const int last = 31 - __clz(hit);
      place = __shfl_sync(0xffffffffu, at, last);
      start = __shfl_sync(0xffffffffu, q, last);
      tokens = __shfl_sync(0xffffffffu, n, last);
    }
    rank += __popc(walked);
  }
  return place;
}
// Heads that the chunks take, others go in turns of four tokens: rows by whole 16-byte copies, d within the block's shared memory.
__host__ inline bool ck_takes(int planes, int d, int dv) { return d % 4 == 0 && dv % 4 == 0 && d <= (planes == CK_GENERAL ? 64 : 128); }
// Columns that U and G have per head: the values' and, with a normaliser, one whose value is 1 and three to fill up.
__host__ __device__ inline int ck_columns(int dv, bool norm) { return norm ? dv + 4 : dv; }
// Floats of the rows, and of U and G, in a workspace.
inline long long ck_work_floats(int planes, int n_tokens, int n_requests, int from, int n_heads, int d, int columns) {
  return d > 128 ? 0 : ck_places(n_tokens, n_requests, from) * n_heads * ck_tile(planes, ck_dmax(d)) + 2LL * n_tokens * n_heads * columns + 8;
}

// The three pieces of two numbers, each pair packed as the operands want it. (Subtractions that the compiler does not draw together
// with the product that made x: the pieces of a number do not depend on what stands around.)
__device__ __forceinline__ void ck_rest(float x, float y, uint32_t pieces, float& rx, float& ry) {
  rx = __fsub_rn(x, __uint_as_float(pieces << 16));
  ry = __fsub_rn(y, __uint_as_float(pieces & 0xffff0000u));
}
__device__ __forceinline__ void ck_split(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(x, y);
  ck_rest(x, y, h, x, y);
  m = pack_bf16(x, y);
  ck_rest(x, y, m, x, y);
  l = pack_bf16(x, y);
}
// The same for any numbers. An infinite one, and one that bfloat16 rounds to infinity, has no second piece: a number near the end of
// the range starts from the largest bfloat16 instead, an infinite one is its first piece and zeros. A product with an infinite
// operand is then right in its first sum alone (the others hold zero times infinity), which `ck_sum` knows.
__device__ __forceinline__ void ck_split_any(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  auto infinite = [](float v) { return (__float_as_uint(v) & 0x7fffffffu) == 0x7f800000u; };
  h = pack_bf16(x, y);
  if ((h & 0x7fffu) == 0x7f80u && !infinite(x)) h -= 1u;
  if ((h & 0x7fff0000u) == 0x7f800000u && !infinite(y)) h -= 0x10000u;
  float rx, ry;
  ck_rest(x, y, h, rx, ry);
  if (infinite(x)) rx = 0.f;
  if (infinite(y)) ry = 0.f;
  m = pack_bf16(rx, ry);
  ck_rest(rx, ry, m, rx, ry);
  l = pack_bf16(rx, ry);
}
// Numbers from 2^60 on, and those that are not finite, are looked for where they enter: a product of two smaller ones, and a state
// that such products are written to sixteen times, stays far from the end of the range. The kernels run as if there were none, and a
// block that has met one does all of its work once more with CAREFUL, which makes the same of every other number. (Looking costs one
// to three per cent of a walk; care inside its loop, with a branch for every pair of numbers, cost a fifth.)
constexpr float CK_LARGE = 1152921504606846976.f;
struct CkLook {      // first pieces: one instruction a pair
  __nv_bfloat162 most = __floats2bfloat162_rn(0.f, 0.f);
  __device__ __forceinline__ void at(const uint32_t (&first)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) most = __hmax2_nan(most, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&first[i])));
  }
  __device__ __forceinline__ bool found() const { return !(__low2float(most) < CK_LARGE && __high2float(most) < CK_LARGE); }
};
// The sum of a product's parts where operands may be infinite.
__device__ __forceinline__ float ck_sum(float hi, float lo) {
  const float s = hi + lo;
  return s == s ? s : hi;
}
__device__ __forceinline__ void stmatrix_x4(void* row, const uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};\n"
               ::"r"(smem_addr(row)), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// hi += a0 b0, lo += the five smaller products, for 2 R tiles of eight: R row blocks of b. Product by product over the tiles: a sum
// waits 21 cycles for the one before it, and the tiles' sums do not depend on one another.
template <int R>
__device__ __forceinline__ void ck_mma(float (&hi)[2 * R][4], float (&lo)[2 * R][4], const uint32_t (&a)[3][4], const uint32_t (&b)[R][3][4]) {
  constexpr int X[6] = {2, 0, 0, 1, 1, 0}, Y[6] = {0, 0, 2, 1, 0, 1};      // the second one: x0 y0
#pragma unroll
  for (int m = 0; m < 6; ++m)
#pragma unroll
    for (int i = 0; i < 2 * R; ++i)
      mma_bf16_16816(m == 1 ? hi[i] : lo[i], a[X[m]], b[i / 2][Y[m]][i % 2 * 2], b[i / 2][Y[m]][i % 2 * 2 + 1]);
}
template <int N>
__device__ __forceinline__ void ck_zero(float (&x)[N][4]) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i][0] = x[i][1] = x[i][2] = x[i][3] = 0.f;
}

// Entry e of what a lane holds of an operand's sixteen tokens and sixteen channels (columns).
__device__ __forceinline__ int ck_token(int lane, int e) { return 2 * (lane & 3) + (e & 1) + 8 * (e >> 2); }
__device__ __forceinline__ int ck_channel(int lane, int e) { return (lane >> 2) + 8 * (e >> 1 & 1); }
__device__ __forceinline__ void ck_operand(const float (&x)[8], uint32_t (&a)[3][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) ck_split(x[2 * i], x[2 * i + 1], a[0][i], a[1][i], a[2][i]);
}
__device__ __forceinline__ void ck_operand_any(const float (&x)[8], uint32_t (&a)[3][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) ck_split_any(x[2 * i], x[2 * i + 1], a[0][i], a[1][i], a[2][i]);
}
template <bool CAREFUL>
__device__ __forceinline__ void ck_operand_of(const float (&x)[8], uint32_t (&a)[3][4], CkLook& look) {
  if (CAREFUL) {
    ck_operand_any(x, a);
  } else {
    ck_operand(x, a);
    look.at(a[0]);
  }
}

struct ChunkArgs {
  const float* tiles;          // [places, heads, ck_tile]
  const float *u, *g;          // [tokens, heads * ck_columns]
  const float* v;              // GENERAL: [tokens, heads * dv]
  float* state;                // [slots, heads, d, dv]
  float* norm_state;           // [slots, heads, d] or null: one more column whose value is 1
  float *o_raw, *nq;           // [tokens, heads * dv], [tokens, heads]
  const int *q_start, *n_new, *slot_ids;
  int n_heads, d, dv, columns;
  int from;                    // requests of fewer tokens are not walked here
};

// The block's shared memory, in floats: stages (a tile, then U, G and V [16][20]), two buffers of the state's pieces [3][16][dmax + 8], the sums of
// the warps that walk [4][16][24] and of those that read [4][16][18].
__host__ __device__ constexpr int ck_stage(int planes, int dmax) { return ck_tile(planes, dmax) + (planes == CK_GENERAL ? 3 : 2) * CK * 20; }
__host__ __device__ constexpr int ck_smem(int planes, int dmax) {
  return 4 * (CK_STAGES * ck_stage(planes, dmax) + 2 * ck_rows(1, dmax) + CK_WARPS * CK_COLS * (24 + 18));
}

// True where the block has to do it again, CAREFUL: nothing of the state is written then.
template <int PLANES, int DMAX, bool CAREFUL>
__device__ __forceinline__ bool state_chunks_of(const ChunkArgs& p, int col_blocks, float* ck_smem_raw) {
  constexpr int CH = DMAX / CK_WARPS, NT = CH / 8, KS = CH / 16, ROW = DMAX + 8, PLANE = 3 * CK * ROW, HALF = 32 * CK_WARPS;
  constexpr int TILE = ck_tile(PLANES, DMAX), STAGE = ck_stage(PLANES, DMAX), VALUES = PLANES == CK_GENERAL ? 3 : 2;
  constexpr bool SYSTEM = PLANES != CK_LINEAR;
  float* stages = ck_smem_raw;
  __nv_bfloat16* held = reinterpret_cast<__nv_bfloat16*>(stages + CK_STAGES * STAGE);      // the state's pieces
  float* sums = stages + CK_STAGES * STAGE + 2 * ck_rows(1, DMAX);
  float* reads = sums + CK_WARPS * CK_COLS * 24;
  // A request's blocks follow one another: the blocks of a long portion then start together, an SM each.
  const int req = blockIdx.x / (col_blocks * p.n_heads), head = blockIdx.x / col_blocks % p.n_heads;
  const int col0 = blockIdx.x % col_blocks * CK_COLS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = p.n_new[req], t0 = p.q_start[req], d = p.d, dv = p.dv, columns = p.columns;
  if (n <= 0 || n < p.from) return false;
  auto sum_of = [](float hi, float lo) { return CAREFUL ? ck_sum(hi, lo) : hi + lo; };
  const int n_chunks = (n + CK - 1) / CK;
  for (int e = tid; e < CK_STAGES * VALUES * CK * 20; e += CK_THREADS)      // columns beyond the values stay 0
    stages[e / (VALUES * CK * 20) * STAGE + TILE + e % (VALUES * CK * 20)] = 0.f;
  __syncthreads();
  // ldmatrix addresses: two tiles of eight tokens (columns, for an operand on the left); of eight channels.
  const int row_plain = (lane & 7) + ((lane >> 4) << 3), col_plain = (lane >> 3 & 1) * 8;
  const int row_trans = (lane & 7) + ((lane >> 3 & 1) << 3), col_trans = (lane >> 4) * 8;
  const int g = lane >> 2, t = lane & 3;

  if (warp >= 2 * CK_WARPS) {
    // The warps that copy.
    const int ct = tid - 2 * HALF, place0 = ck_place(t0, ck_rank(p.n_new, req, p.from));
    auto load = [&](int chunk) {
      if (chunk < n_chunks) {
        float* to = stages + chunk % CK_STAGES * STAGE;
        const float* tile = p.tiles + ((size_t)(place0 + chunk) * p.n_heads + head) * TILE;
#pragma unroll 4
        for (int e = ct; e < TILE / 4; e += HALF) cp_async_16(to + 4 * e, tile + 4 * e, 16);
        const int at = ct >> 2, piece = col0 + (ct & 3) * 4, token = chunk * CK + at;
        if (ct < CK * 4 && piece < columns) {
          to += TILE + at * 20 + (ct & 3) * 4;
          const bool there = token < n;
          const size_t from = ((size_t)(t0 + (there ? token : 0)) * p.n_heads + head) * columns + piece;
          cp_async_16(to, p.u + from, there ? 16 : 0);
          cp_async_16(to + CK * 20, p.g + from, there ? 16 : 0);
          if (PLANES == CK_GENERAL) cp_async_16(to + 2 * CK * 20, p.v + from, there ? 16 : 0);      // (columns = dv)
        }
      }
      cp_async_commit();
    };
    load(0);
    load(1);
    cp_async_wait<1>();
    __syncthreads();
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
      load(chunk + 2);      // in the place of chunk - 2, which everyone has left
      cp_async_wait<1>();
      __syncthreads();
    }
    cp_async_wait<0>();
    return !CAREFUL && __syncthreads_or(0);
  }
  if (warp >= CK_WARPS) {
    // The warps that read out.
    const int ct = tid - HALF, ch0 = (warp - CK_WARPS) * CH;
    auto read_out = [&](int chunk) {
      const float* base = stages + chunk % CK_STAGES * STAGE;
      const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(base);
      uint32_t b[KS][3][4];
#pragma unroll
      for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int x = 0; x < 3; ++x)
          ldmatrix_x4(b[ks][x], rows + CK_F * PLANE + (x * CK + row_plain) * ROW + ch0 + 16 * ks + col_plain);
      float hi[2][4], lo[2][4];
      ck_zero(hi);
      ck_zero(lo);
      const __nv_bfloat16* state = held + (chunk & 1) * PLANE;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t a[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) ldmatrix_x4(a[x], state + (x * CK + row_trans) * ROW + ch0 + 16 * ks + col_trans);
        ck_mma<1>(hi, lo, a, reinterpret_cast<const uint32_t (&)[1][3][4]>(b[ks]));
      }
      float* to = reads + ((warp - CK_WARPS) * CK_COLS + g) * 18 + 2 * t;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          *reinterpret_cast<float2*>(to + c * 8 * 18 + i * 8) = make_float2(sum_of(hi[i][2 * c], lo[i][2 * c]), sum_of(hi[i][2 * c + 1], lo[i][2 * c + 1]));
      __syncwarp();
      asm volatile("bar.sync 2, 128;" ::: "memory");      // every reading warp's sums are there
      const int at = ct >> 3, c = 2 * (ct & 7), col = col0 + c;
      float2 o = *reinterpret_cast<const float2*>(base + TILE + CK * 20 + at * 20 + c);
      float2 s = make_float2(0.f, 0.f);
#pragma unroll
      for (int w = 0; w < CK_WARPS; ++w) {
        s.x += reads[(w * CK_COLS + c) * 18 + at];
        s.y += reads[(w * CK_COLS + c + 1) * 18 + at];
      }
      o.x += s.x;
      o.y += s.y;
      if (chunk * CK + at < n) {
        const size_t token = (size_t)(t0 + chunk * CK + at) * p.n_heads + head;
        if (col < dv) *reinterpret_cast<float2*>(p.o_raw + token * dv + col) = o;      // (dv and col are even)
        else if (col == dv && p.norm_state) p.nq[token] = o.x;
      }
    };
    __syncthreads();
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
      if (chunk > 0) read_out(chunk - 1);      // while the next one is walked
      __syncthreads();
    }
    read_out(n_chunks - 1);
    return !CAREFUL && __syncthreads_or(0);
  }

  // The warps that walk. Lane 4 g + t: columns g and g + 8.
  const int ch0 = warp * CH;
  const size_t slot = (size_t)p.slot_ids[req];
  float* S_g = p.state + (slot * p.n_heads + head) * (size_t)d * dv;
  float* N_g = p.norm_state ? p.norm_state + (slot * p.n_heads + head) * (size_t)d : nullptr;
  float S[NT][4];      // entry e of a tile: column g + 8 (e >> 1), channel ch0 + 8 tile + 2 t + (e & 1)
  auto state_at = [&](int nt, int e) -> float* {
    const int ch = ch0 + 8 * nt + 2 * t + (e & 1), col = col0 + g + 8 * (e >> 1);
    if (ch >= d) return nullptr;
    return col < dv ? S_g + (size_t)ch * dv + col : (N_g && col == dv ? N_g + ch : nullptr);
  };
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float* at = state_at(nt, e);
      S[nt][e] = at ? *at : 0.f;
    }
  CkLook look;
  int large = 0;
  __syncthreads();      // chunk 0

  for (int chunk = 0; chunk < n_chunks; ++chunk) {
    const float* base = stages + chunk % CK_STAGES * STAGE;
    const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(base);
    // The state's pieces, for W S here and for the read-outs.
    uint32_t a[KS][3][4];
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float s0 = S[2 * ks + (i >> 1)][2 * (i & 1)], s1 = S[2 * ks + (i >> 1)][2 * (i & 1) + 1];
        if (CAREFUL) ck_split_any(s0, s1, a[ks][0][i], a[ks][1][i], a[ks][2][i]);
        else ck_split(s0, s1, a[ks][0][i], a[ks][1][i], a[ks][2][i]);
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) stmatrix_x4(held + (chunk & 1) * PLANE + (x * CK + row_trans) * ROW + ch0 + 16 * ks + col_trans, a[ks][x]);
      look.at(a[ks][0]);
    }
    large |= __float_as_int(base[ck_flag(DMAX)]);
    // Entry e of what a column's tokens bring, in the order of an operand: token 2 t + (e & 1) + 8 (e >> 2) of column
    // g + 8 (e >> 1 & 1).
    auto values = [&](int which, float (&v)[8]) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = base[TILE + which * CK * 20 + (2 * t + (e & 1) + 8 * (e >> 2)) * 20 + g + 8 * (e >> 1 & 1)];
    };
    // What the chunk writes into the state.
    float add[NT][4], add_lo[NT][4];
    ck_zero(add);
    ck_zero(add_lo);
    uint32_t written[NT / 2][3][4];
    auto written_rows = [&](int plane) {
#pragma unroll
      for (int np = 0; np < NT / 2; ++np)
#pragma unroll
        for (int x = 0; x < 3; ++x)
          ldmatrix_x4_trans(written[np][x], rows + plane * PLANE + (x * CK + row_trans) * ROW + ch0 + 16 * np + col_trans);
    };
    auto write = [&](const float (&what)[8]) {
      uint32_t left[3][4];
      if (CAREFUL) ck_operand_any(what, left);
      else ck_operand(what, left);
      ck_mma<NT / 2>(add, add_lo, left, written);
    };
    if constexpr (PLANES == CK_GENERAL) {
      float v[8];
      values(2, v);
      written_rows(CK_C);
      write(v);
    }
    written_rows(CK_B);      // (ahead of the exchange)
    float y[8];
    values(0, y);
    if constexpr (SYSTEM) {
      float hi[2][4], lo[2][4];
      ck_zero(hi);
      ck_zero(lo);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t b[1][3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x)
          ldmatrix_x4(b[0][x], rows + CK_W * PLANE + (x * CK + row_plain) * ROW + ch0 + 16 * ks + col_plain);
        ck_mma<1>(hi, lo, a[ks], b);
      }
      float* to = sums + (warp * CK_COLS + g) * 24 + 2 * t;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          *reinterpret_cast<float2*>(to + c * 8 * 24 + i * 8) = make_float2(sum_of(hi[i][2 * c], lo[i][2 * c]), sum_of(hi[i][2 * c + 1], lo[i][2 * c + 1]));
      __syncwarp();
      asm volatile("bar.sync 1, 128;" ::: "memory");      // every walking warp's sums are there
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 s[CK_WARPS];
#pragma unroll
        for (int w = 0; w < CK_WARPS; ++w)
          s[w] = *reinterpret_cast<const float2*>(sums + (w * CK_COLS + g + 8 * (i & 1)) * 24 + 8 * (i >> 1) + 2 * t);
        y[2 * i] += (s[0].x + s[1].x) + (s[2].x + s[3].x);
        y[2 * i + 1] += (s[0].y + s[1].y) + (s[2].y + s[3].y);
      }
    }
    if (CAREFUL)      // tokens beyond the last one write nothing (their rows are zeros, and zero times infinity is no number)
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (chunk * CK + ck_token(lane, e) >= n) y[e] = 0.f;
    write(y);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float2 decay = *reinterpret_cast<const float2*>(base + ck_rows(PLANES, DMAX) + ch0 + 8 * i + 2 * t);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float written_here = !CAREFUL || ch0 + 8 * i + 2 * t + (e & 1) < d ? sum_of(add[i][e], add_lo[i][e]) : 0.f;      // (nor do channels beyond d)
        S[i][e] = fmaf(e & 1 ? decay.y : decay.x, S[i][e], written_here);
      }
    }
    __syncthreads();      // the next chunk is there, and everyone is done with this one
  }
  if (!CAREFUL && __syncthreads_or(large || look.found())) return true;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float* at = state_at(nt, e);
      if (at) *at = S[nt][e];
    }
  return false;
}
template <int PLANES, int DMAX>
__device__ __noinline__ void state_chunks_carefully(const ChunkArgs& p, int col_blocks, float* smem) {
  state_chunks_of<PLANES, DMAX, true>(p, col_blocks, smem);
}
template <int PLANES, int DMAX>
__global__ void __launch_bounds__(CK_THREADS, 2 * ck_smem(PLANES, DMAX) <= 226 * 1024 ? 2 : 1)
state_chunks_kernel(const __grid_constant__ ChunkArgs p, int col_blocks) {
  extern __shared__ __align__(16) float ck_smem_raw[];
  if (state_chunks_of<PLANES, DMAX, false>(p, col_blocks, ck_smem_raw)) state_chunks_carefully<PLANES, DMAX>(p, col_blocks, ck_smem_raw);
}

template <int PLANES, int DMAX>
static int launch_state_chunks_of(const ChunkArgs& a, int n_requests, cudaStream_t stream) {
  constexpr size_t smem = ck_smem(PLANES, DMAX);
  static_assert(smem <= 227 * 1024, "the block's shared memory");
  cudaError_t e = cudaFuncSetAttribute(state_chunks_kernel<PLANES, DMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return llmrs_fail("state chunks: shared memory %zu: %s", smem, cudaGetErrorString(e));
  const int col_blocks = (a.dv + (a.norm_state ? 1 : 0) + CK_COLS - 1) / CK_COLS;
  const long long blocks = (long long)n_requests * a.n_heads * col_blocks;
  LLMRS_REQUIRE(blocks <= 0x7fffffffLL, "state chunks: too many requests, heads or columns");
  state_chunks_kernel<PLANES, DMAX><<<(unsigned)blocks, CK_THREADS, smem, stream>>>(a, col_blocks);
  return llmrs_launch_status("state chunks");
}
template <int PLANES>
static int launch_state_chunks(const ChunkArgs& a, int n_requests, cudaStream_t stream) {
  if (PLANES == CK_GENERAL || a.d <= 64) return launch_state_chunks_of<PLANES, 64>(a, n_requests, stream);
  return launch_state_chunks_of<PLANES, PLANES == CK_GENERAL ? 64 : 128>(a, n_requests, stream);
}

// ---- rows ------------------------------------------------------------------------------------------------------------
// The products over tokens run transposed on the tensor cores, sixteen channels (or value columns) a warp: entry e of what a lane
// 4 g + t holds of them is token 2 t + (e & 1) + 8 (e >> 2) of channel g + 8 (e >> 1 & 1) (`ck_token`, `ck_channel`), the order of an
// operand and, as it happens, of the sums that come out.
// A matrix over the chunk's tokens in shared memory, [3][16][24]: three pieces, rows of 48 bytes (no two of eight on the same banks).
// What lies above the diagonal must be zero.
constexpr int CK_MATRIX = 3 * CK * 24;
template <bool CAREFUL>
__device__ __forceinline__ void ck_set(__nv_bfloat16* m, int i, int j, float x) {
  uint32_t piece[3];
  if (CAREFUL) ck_split_any(x, 0.f, piece[0], piece[1], piece[2]);
  else ck_split(x, 0.f, piece[0], piece[1], piece[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) m[(k * CK + i) * 24 + j] = __ushort_as_bfloat16((unsigned short)piece[k]);
}
// out[token i] += sum_j m[i][j] x[token j]. CAREFUL: an x that is not finite reaches the tokens from its own on and no earlier one:
// zero times it would be no number, so it goes in as zero and its products are added by themselves.
template <bool CAREFUL>
__device__ __forceinline__ void ck_apply(const __nv_bfloat16* m, const float (&x)[8], int lane, float (&out)[8], CkLook& look) {
  auto finite = [](float v) { return (__float_as_uint(v) & 0x7fffffffu) < 0x7f800000u; };
  float hi[2][4], lo[2][4];
  uint32_t a[3][4], b[1][3][4];
  ck_zero(hi);
  ck_zero(lo);
#pragma unroll
  for (int k = 0; k < 3; ++k) ldmatrix_x4(b[0][k], m + (k * CK + (lane & 7) + ((lane >> 4) << 3)) * 24 + (lane >> 3 & 1) * 8);
  if constexpr (!CAREFUL) {
    ck_operand(x, a);
    look.at(a[0]);
    look.at(b[0][0]);
    ck_mma<1>(hi, lo, a, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) out[e] += hi[e >> 2][e & 3] + lo[e >> 2][e & 3];
  } else {
    float y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = finite(x[e]) ? x[e] : 0.f;
    ck_operand_any(y, a);
    ck_mma<1>(hi, lo, a, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) out[e] += ck_sum(hi[e >> 2][e & 3], lo[e >> 2][e & 3]);
#pragma unroll
    for (int j = 0; j < CK; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {      // token j of the lane's channel c: lane j % 8 / 2 of its four has it
        const float xj = __shfl_sync(0xffffffffu, x[(j & 1) + 2 * c + 4 * (j >> 3)], (lane & ~3) | (j & 7) >> 1);
        if (!finite(xj)) {
#pragma unroll
          for (int e = 2 * c; e < 8; e += (e & 1) ? 3 : 1) {
            const int i = ck_token(lane, e);
            const __nv_bfloat16* at = m + i * 24 + j;
            if (i >= j) out[e] = fmaf((__bfloat162float(at[0]) + __bfloat162float(at[CK * 24])) + __bfloat162float(at[2 * CK * 24]), xj, out[e]);
          }
        }
        __syncwarp();
      }
  }
}
// Rows of a plane, channels c0 .. c0 + 15.
__device__ __forceinline__ void ck_put(float* tile, int plane, int row, int c0, int lane, const uint32_t (&a)[3][4]) {
  __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(tile) + (plane * 3 * CK + (lane & 7) + ((lane >> 4) << 3)) * row + c0 + (lane >> 3 & 1) * 8;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};\n"
                 ::"r"(smem_addr(to + k * CK * row)), "r"(a[k][0]), "r"(a[k][1]), "r"(a[k][2]), "r"(a[k][3]) : "memory");
}
// W = T x into its plane, then f + Q W, F.
template <bool CAREFUL>
__device__ __forceinline__ void ck_system_rows(float* tile, int plane, int row, int c0, int lane, const __nv_bfloat16* T, const __nv_bfloat16* Q,
                                               const float (&x)[8], float (&f)[8], CkLook& look) {
  uint32_t a[3][4];
  float w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = 0.f;
  ck_apply<CAREFUL>(T, x, lane, w, look);
  ck_operand_of<CAREFUL>(w, a, look);
  ck_put(tile, plane, row, c0, lane, a);
  ck_apply<CAREFUL>(Q, w, lane, f, look);
}
// Column c of (I + sign M)^-1 diag(scale), M below the diagonal with rows `stride` apart: forward substitution.
template <bool CAREFUL>
__device__ __forceinline__ void ck_solve(const float* m, int stride, float sign, int c, float scale, __nv_bfloat16* out) {
  float col[CK];
#pragma unroll
  for (int i = 0; i < CK; ++i) {
    float acc = i == c ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < i; ++j) acc = fmaf(-sign * m[i * stride + j], col[j], acc);
    col[i] = i >= c ? acc : 0.f;      // (what is no number in a row of M stays in the rows from it on)
    ck_set<CAREFUL>(out, i, c, i >= c ? acc * scale : 0.f);
  }
}
// hi + lo times x, lo being what rounding took from hi.
__device__ __forceinline__ void ck_times(float& hi, float& lo, float x) {
  const float product = __fmul_rn(hi, x);
  lo = fmaf(lo, x, fmaf(hi, x, -product));
  hi = product;
}

struct ChunkRowsArgs {
  const float *q, *k;          // [tokens, stride], group's channels at group * d
  long long stride;
  const float* v;              // [tokens, heads * dv]
  const float *decay, *head_decay;      // [tokens, heads] or null (then [heads], or 1)
  const float* beta;           // [tokens, heads] or null (1): write strengths, without a system gains
  const float* skip;           // [heads] or null (0)
  const int *q_start, *n_new;
  float *tiles, *u, *g;
  int n_requests, n_heads, n_groups, d, dv, columns, from;
  int heads_a_block;           // of the heads that share a key head (the launch sets it)
  bool norm;
};

// A tile is put together in shared memory and leaves by one bulk copy. Every thread that wrote to it calls ck_tile_written before a
// barrier, one thread ck_tile_leaves after it, and ck_tile_left before the tile is written again or the block ends.
__device__ __forceinline__ void ck_tile_written() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void ck_tile_leaves(float* to, const float* tile, int floats) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;"
               ::"l"(to), "r"(smem_addr(tile)), "r"(floats * 4) : "memory");
}
__device__ __forceinline__ void ck_tile_left() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// All threads, before the block's tiles are made once more: the first ones (of thread 0) are in memory.
__device__ __forceinline__ void ck_tile_again() {
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();
}

// The rows of CK_LINEAR and CK_SYSTEM with a decay per token and head: a block per (place, key head, some of the heads that share it).
// First the products of the rows on the tensor cores, a quarter of the channels a warp; then, two heads at a time, the coefficients (a
// warp a head); then head by head the rows, sixteen channels and sixteen columns a warp at a time. Bound by memory latency and the
// bytes that leave (39 KB a chunk and head of 128 channels): 2,048 tokens of 16 heads over 8 of 128 x 128 47 us (two channels a thread
// and products on the CUDA cores 61), 16 heads without a system 39. Three blocks an SM: with two, the products apart from the
// tile, 55 and 48. Heads that share one key head by a block each pair: a Mamba-2 mixer of 32 heads over one group, 64 tokens
// 128 us, 186 with all of them in one block; 2,048 tokens 1,628 and 1,645.
constexpr int CK_ROWS_THREADS = 256;
__host__ __device__ constexpr int ck_rows_smem(int planes, int dmax) { return 4 * (ck_tile(planes, dmax) + 2 * CK * (dmax + 4)); }
struct CkRowsShared {      // beside the tile
  float gram[2][CK][CK + 1], strengths[2][2][CK], P[2][CK], Z[2][CK], own[2][CK][CK + 1];
  alignas(16) __nv_bfloat16 Q[2][CK_MATRIX], T[2][CK_MATRIX];
};
// True where CAREFUL would make something else of it.
template <int PLANES, int DMAX, bool CAREFUL>
__device__ __forceinline__ bool ck_rows_of(const ChunkRowsArgs& p, float* tile, CkRowsShared& sh) {
  constexpr int RS = DMAX + 4, GS = CK + 1, ROW = DMAX + 8, THREADS = CK_ROWS_THREADS, HEADS = 2, WARPS = 4;
  constexpr int EACH = (2 * CK * (DMAX / 4) + THREADS - 1) / THREADS;
  constexpr bool SYSTEM = PLANES == CK_SYSTEM;
  float* rows = tile + ck_tile(PLANES, DMAX);      // k, q: [2][16][RS]
  auto part = reinterpret_cast<float (*)[2][CK][CK]>(tile);      // [WARPS]: a warp's share of the products, before there is a tile
  static_assert(ck_tile(PLANES, DMAX) >= WARPS * 2 * CK * CK, "the products lie where the tile will be");
  auto& gram = sh.gram;
  auto& strengths = sh.strengths;
  auto& P = sh.P;
  auto& Z = sh.Z;
  auto& own = sh.own;
  auto& Q = sh.Q;
  auto& T = sh.T;
  CkLook look;
  const int place = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = p.d;
  const int shared = p.n_heads / p.n_groups, parts = (shared + p.heads_a_block - 1) / p.heads_a_block, group = blockIdx.y / parts;
  const int head0 = group * shared + blockIdx.y % parts * p.heads_a_block, head1 = min(head0 + p.heads_a_block, (group + 1) * shared);
  int t_req, n_req;
  const int place0 = ck_request(p.q_start, p.n_new, p.n_requests, p.from, place, t_req, n_req);
  const int first = (place - place0) * CK, have = min(CK, n_req - first);
  if (first < 0 || have <= 0 || n_req < p.from) return false;
  const size_t t0 = (size_t)(t_req + first);
  float decay_in = 0.f, beta_in = 0.f;      // of token `lane` and this warp's head, the first ones on their way early
  auto fetch_strengths = [&](int h, float& decay, float& beta) {
    const size_t at = (t0 + lane) * p.n_heads + h;
    decay = lane >= have ? 1.f : (p.decay ? p.decay[at] : (p.head_decay ? p.head_decay[h] : 1.f));
    beta = lane >= have ? 0.f : (p.beta ? p.beta[at] : 1.f);
  };
  if (warp < min(HEADS, head1 - head0)) fetch_strengths(head0 + warp, decay_in, beta_in);
  {
    float4 in[EACH];
#pragma unroll
    for (int x = 0; x < EACH; ++x) {
      const int e = tid + x * THREADS, a = e / (CK * (DMAX / 4)), t = e / (DMAX / 4) % CK, c = e % (DMAX / 4) * 4;
      in[x] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a < 2 && t < have && c < d)
        in[x] = __ldg(reinterpret_cast<const float4*>((a ? p.q : p.k) + (t0 + t) * p.stride + (size_t)group * d + c));
    }
#pragma unroll
    for (int x = 0; x < EACH; ++x) {
      const int e = tid + x * THREADS;
      if (e < 2 * CK * (DMAX / 4)) *reinterpret_cast<float4*>(rows + e / (DMAX / 4) * RS + e % (DMAX / 4) * 4) = in[x];
    }
  }
  __syncthreads();
  if (warp < WARPS) {
    const int g = lane >> 2, t = lane & 3;
    float hi[2][2][4], lo[2][2][4];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      ck_zero(hi[a]);
      ck_zero(lo[a]);
    }
#pragma unroll
    for (int ks = 0; ks < DMAX / 16 / WARPS; ++ks) {
      const int c = (warp * (DMAX / 16 / WARPS) + ks) * 16 + 2 * t;
      uint32_t left[2][3][4], right[1][3][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = *reinterpret_cast<const float2*>(rows + (a * CK + g + 8 * (i & 1)) * RS + c + 8 * (i >> 1));
          if (CAREFUL) ck_split_any(x.x, x.y, left[a][0][i], left[a][1][i], left[a][2][i]);
          else ck_split(x.x, x.y, left[a][0][i], left[a][1][i], left[a][2][i]);
        }
      look.at(left[0][0]);
      look.at(left[1][0]);
#pragma unroll
      for (int x = 0; x < 3; ++x) {      // k on the right: tokens g, then g + 8, of both halves of the channels
        right[0][x][0] = left[0][x][0];
        right[0][x][1] = left[0][x][2];
        right[0][x][2] = left[0][x][1];
        right[0][x][3] = left[0][x][3];
      }
      if (SYSTEM) ck_mma<1>(hi[0], lo[0], left[0], right);
      ck_mma<1>(hi[1], lo[1], left[1], right);
    }
#pragma unroll
    for (int a = SYSTEM ? 0 : 1; a < 2; ++a)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[warp][a][g + 8 * (e >> 1)][8 * i + 2 * t + (e & 1)] = CAREFUL ? ck_sum(hi[a][i][e], lo[a][i][e]) : hi[a][i][e] + lo[a][i][e];
  }
  __syncthreads();
  for (int e = tid; e < 2 * CK * CK; e += THREADS) {
    const int a = e / (CK * CK), i = e / CK % CK, j = e % CK;
    if (SYSTEM || a) gram[a][i][j] = (part[0][a][i][j] + part[1][a][i][j]) + (part[2][a][i][j] + part[3][a][i][j]);
  }
  for (int h0 = head0; h0 < head1; h0 += HEADS) {
    const int heads = min(HEADS, head1 - h0);
    __syncthreads();      // the products; everyone is done with the heads before
    if (warp < heads) {
      if (h0 > head0) fetch_strengths(h0 + warp, decay_in, beta_in);
      if (lane < CK) {
        const int i = lane;
        strengths[warp][0][i] = decay_in;
        strengths[warp][1][i] = beta_in;
        __syncwarp(0xffffu);
        // The decays after j up to and with i; after i. Each product with what rounding took from it: a decay that all tokens share
        // would otherwise be off by the same sixteen roundings in every chunk.
        float between = 1.f, between_lo = 0.f, after = 1.f, after_lo = 0.f;
#pragma unroll
        for (int j = CK - 1; j >= 0; --j) {
          const float decay = strengths[warp][0][j], w = __fadd_rn(between, between_lo);
          ck_set<CAREFUL>(Q[warp], i, j, j <= i ? gram[1][i][j] * w : 0.f);
          if (SYSTEM && j < i) own[warp][i][j] = beta_in * (gram[0][i][j] * w);
          if (j <= i) ck_times(between, between_lo, decay);
          if (j > i) ck_times(after, after_lo, decay);
        }
        P[warp][i] = __fadd_rn(between, between_lo);
        Z[warp][i] = __fadd_rn(after, after_lo);
        __syncwarp(0xffffu);
        if (SYSTEM) ck_solve<CAREFUL>(&own[warp][0][0], GS, 1.f, i, beta_in, T[warp]);
      }
    }
    for (int x = 0; x < heads; ++x) {
      const int h = h0 + x;
      // The values that this warp needs below are on their way while it makes its channels' rows.
      const int groups = (p.columns + 15) / 16;
      float v[8];
      auto fetch = [&](int group) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int at = ck_token(lane, e), col = 16 * group + ck_channel(lane, e);
          v[e] = p.norm && col == p.dv ? 1.f : 0.f;
          if (at < have && col < p.dv) v[e] = __ldg(p.v + ((t0 + at) * p.n_heads + h) * p.dv + col);
        }
      };
      if (warp < groups) fetch(warp);
      if (tid == 0) {
        ck_tile_left();
        tile[ck_flag(DMAX)] = __int_as_float(CAREFUL);
      }
      __syncthreads();      // the coefficients; the tile before has left
      float before[8], after[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        before[e] = P[x][ck_token(lane, e)];
        after[e] = Z[x][ck_token(lane, e)];
      }
      for (int c0 = 16 * warp; c0 < DMAX; c0 += 16 * (THREADS / 32)) {
        uint32_t a[3][4];
        float k[8], q[8], f[8], out[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float* at = rows + ck_token(lane, e) * RS + c0 + ck_channel(lane, e);
          k[e] = at[0];
          q[e] = at[CK * RS];
          f[e] = 0.f;
        }
        if constexpr (SYSTEM) {
#pragma unroll
          for (int e = 0; e < 8; ++e) out[e] = -before[e] * k[e];
          ck_system_rows<CAREFUL>(tile, CK_W, ROW, c0, lane, T[x], Q[x], out, f, look);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = fmaf(before[e], q[e], f[e]);
        ck_operand_of<CAREFUL>(f, a, look);
        ck_put(tile, CK_F, ROW, c0, lane, a);
#pragma unroll
        for (int e = 0; e < 8; ++e) out[e] = after[e] * k[e];
        ck_operand_of<CAREFUL>(out, a, look);
        ck_put(tile, CK_B, ROW, c0, lane, a);
        if (lane < 16) tile[ck_rows(PLANES, DMAX) + c0 + lane] = P[x][CK - 1];
      }
      ck_tile_written();
      for (int group = warp; group < groups; group += THREADS / 32) {
        if (group != warp) fetch(group);
        const float skip = p.skip ? p.skip[h] : 0.f;
        float u[8], g[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          g[e] = 0.f;
          u[e] = SYSTEM ? 0.f : strengths[x][1][ck_token(lane, e)] * v[e];
        }
        if constexpr (SYSTEM) ck_apply<CAREFUL>(T[x], v, lane, u, look);
        ck_apply<CAREFUL>(Q[x], u, lane, g, look);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int at = ck_token(lane, e), col = 16 * group + ck_channel(lane, e);
          if (at < have && col < p.columns) {
            const size_t to = ((t0 + at) * p.n_heads + h) * p.columns + col;
            p.u[to] = u[e];
            p.g[to] = skip == 0.f ? g[e] : fmaf(skip, v[e], g[e]);
          }
        }
      }
      __syncthreads();
      if (tid == 0) ck_tile_leaves(p.tiles + ((size_t)place * p.n_heads + h) * ck_tile(PLANES, DMAX), tile, ck_tile(PLANES, DMAX));
    }
  }
  if (tid == 0) ck_tile_left();
  return !CAREFUL && look.found();
}
template <int PLANES, int DMAX>
__device__ __noinline__ void ck_rows_carefully(const ChunkRowsArgs& p, float* tile, CkRowsShared& sh) {
  ck_tile_again();
  ck_rows_of<PLANES, DMAX, true>(p, tile, sh);
}
template <int PLANES, int DMAX>
__global__ void __launch_bounds__(CK_ROWS_THREADS, 3)
ck_rows_kernel(const __grid_constant__ ChunkRowsArgs p) {
  extern __shared__ __align__(128) float ck_rows_raw[];
  __shared__ CkRowsShared sh;
  if (__syncthreads_or(ck_rows_of<PLANES, DMAX, false>(p, ck_rows_raw, sh))) ck_rows_carefully<PLANES, DMAX>(p, ck_rows_raw, sh);
}

template <int PLANES, int DMAX>
static int launch_ck_rows_of(const ChunkRowsArgs& p, dim3 grid, cudaStream_t stream) {
  constexpr size_t smem = ck_rows_smem(PLANES, DMAX);
  if (smem > 32 * 1024) {      // (48 KB need no asking, but the kernel's own 14 KB count too)
    cudaError_t e = cudaFuncSetAttribute(ck_rows_kernel<PLANES, DMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return llmrs_fail("state chunks: shared memory %zu: %s", smem, cudaGetErrorString(e));
  }
  ck_rows_kernel<PLANES, DMAX><<<grid, CK_ROWS_THREADS, smem, stream>>>(p);
  return llmrs_launch_status("state chunks (rows)");
}
template <int PLANES>
static int launch_ck_rows(ChunkRowsArgs p, int n_tokens, cudaStream_t stream) {
  // Heads that share a key head go through one block, which makes their products once, as long as there are blocks enough: three for
  // each of the SMs, two heads (whose coefficients are made together) at least.
  const long long places = ck_places(n_tokens, p.n_requests, p.from), shared = p.n_heads / p.n_groups, blocks = 3 * 148;
  p.heads_a_block = (int)std::min(shared, std::max(2ll, places * p.n_heads / blocks / 2 * 2));
  const dim3 grid((unsigned)places, (unsigned)(p.n_groups * ((shared + p.heads_a_block - 1) / p.heads_a_block)));
  LLMRS_REQUIRE(grid.y <= 65535, "state chunks: too many heads");
  return p.d <= 64 ? launch_ck_rows_of<PLANES, 64>(p, grid, stream) : launch_ck_rows_of<PLANES, 128>(p, grid, stream);
}
