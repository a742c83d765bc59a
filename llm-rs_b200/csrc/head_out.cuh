// The output stage that the recurrent mixers share: every head's read-out divided by its root mean square, times a weight, times
// SiLU or the sigmoid of a gate, rounded to the activation type. For heads whose channels are a power of two of pieces of four
// (dv 4 to 128): a lane takes one piece with one load of each operand, a head's lanes are neighbours.
// Bound by memory. 2,048 tokens, a warp a head with a load a channel and the head read twice -> this, us: 16 heads of 128
// HO_GATED, with a normaliser (1,793 tokens) HO_LINEAR, 32 heads of 64 HO_DELTA.
#pragma once
#include "common.cuh"
#include "short_conv.cuh"

struct HeadOutArgs {
  const float* o;                   // [tokens, heads * dv]
  const float *nq, *floor_;         // [tokens, heads] or null: o is divided by max(|nq|, floor) + den_eps first
  float den_eps;
  const void* gate;                 // rows gate_stride apart
  long long gate_stride;
  const float* w;                   // [heads * dv], or [dv] with w_shared; null: none
  int w_shared;
  void* out;                        // rows out_stride apart
  long long out_stride;
  int n_tokens, n_heads, dv;
  float eps, out_scale;
  int silu;
};

constexpr int HO_ROWS = 4;      // heads a group of lanes takes, their loads in flight together
template <typename TA>
static __global__ void __launch_bounds__(256) head_out_kernel(const HeadOutArgs a, int lanes) {
  struct alignas(4 * sizeof(TA)) Piece { TA x[4]; };
  const int piece = threadIdx.x & (lanes - 1), n_rows = a.n_tokens * a.n_heads, apart = 256 / lanes;
  const int row0 = blockIdx.x * (HO_ROWS * apart) + threadIdx.x / lanes;
  float4 o[HO_ROWS], w[HO_ROWS];
  Piece gate[HO_ROWS];
  float nq[HO_ROWS], floor_[HO_ROWS];
  int t[HO_ROWS], c[HO_ROWS];
#pragma unroll
  for (int r = 0; r < HO_ROWS; ++r) {      // all loads first
    const int row = min(row0 + r * apart, n_rows - 1);
    t[r] = row / a.n_heads;
    c[r] = (row - t[r] * a.n_heads) * a.dv + piece * 4;
    o[r] = *reinterpret_cast<const float4*>(a.o + (size_t)row * a.dv + piece * 4);
    gate[r] = *reinterpret_cast<const Piece*>(reinterpret_cast<const TA*>(a.gate) + (size_t)t[r] * a.gate_stride + c[r]);
    w[r] = make_float4(1.f, 1.f, 1.f, 1.f);
    if (a.w) w[r] = *reinterpret_cast<const float4*>(a.w + (a.w_shared ? piece * 4 : c[r]));
    if (a.nq) {
      nq[r] = a.nq[row];
      floor_[r] = a.floor_[row];
    }
  }
#pragma unroll
  for (int r = 0; r < HO_ROWS; ++r) {
    if (a.nq) {
      const float id = 1.0f / (fmaxf(fabsf(nq[r]), floor_[r]) + a.den_eps);
      o[r].x *= id; o[r].y *= id; o[r].z *= id; o[r].w *= id;
    }
    float ss = fmaf(o[r].x, o[r].x, fmaf(o[r].y, o[r].y, fmaf(o[r].z, o[r].z, o[r].w * o[r].w)));
    for (int off = lanes / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float inv = 1.0f / sqrtf(ss / (float)a.dv + a.eps) * a.out_scale;
    auto gated = [&](float v, float weight, TA g) {
      const float x = to_float(g);
      return from_float<TA>(v * inv * weight * (a.silu ? rec_silu(x) : rec_sigmoid(x)));
    };
    Piece y;
    y.x[0] = gated(o[r].x, w[r].x, gate[r].x[0]);
    y.x[1] = gated(o[r].y, w[r].y, gate[r].x[1]);
    y.x[2] = gated(o[r].z, w[r].z, gate[r].x[2]);
    y.x[3] = gated(o[r].w, w[r].w, gate[r].x[3]);
    if (row0 + r * apart < n_rows)
      *reinterpret_cast<Piece*>(reinterpret_cast<TA*>(a.out) + (size_t)t[r] * a.out_stride + c[r]) = y;
  }
}

// Whether every piece of four lies on its boundary.
template <typename TA>
static bool head_out_takes(const HeadOutArgs& a) {
  const int lanes = a.dv / 4;
  auto starts = [](const void* p, size_t bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; };
  return a.dv % 4 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && a.gate_stride % 4 == 0 && a.out_stride % 4 == 0 &&
         starts(a.o, 16) && starts(a.w, 16) && starts(a.gate, 4 * sizeof(TA)) && starts(a.out, 4 * sizeof(TA)) &&
         (long long)a.n_tokens * a.n_heads <= 0x7fffffff;
}
template <typename TA>
static void launch_head_out(const HeadOutArgs& a, cudaStream_t stream) {
  const int lanes = a.dv / 4, rows = HO_ROWS * (256 / lanes);
  const long long n_rows = (long long)a.n_tokens * a.n_heads;
  head_out_kernel<TA><<<(unsigned)((n_rows + rows - 1) / rows), 256, 0, stream>>>(a, lanes);
}
