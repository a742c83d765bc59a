// The output stage that the recurrent mixers share: every head's read-out divided by its root mean square, times a weight, times
// SiLU or the sigmoid of a gate, rounded to the activation type. For heads whose channels are a power of two of pieces of four
// (dv 4 to 128): a lane takes one piece with one load of each operand, a head's lanes are neighbours.
// 2,048 tokens, a warp a head with a load a channel and the head read twice -> this, us: 16 heads of 128 15.4 -> 13.2, with a
// normaliser (1,793 tokens) 24.6 -> 12.4, 32 heads of 64 22.2 -> 12.9. Bound by memory's latency (four heads a group of lanes, their
// loads in flight together, cost registers: 14.8, 15.5, 15.8).
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

template <typename TA>
static __global__ void __launch_bounds__(256) head_out_kernel(const HeadOutArgs a, int lanes) {
  struct alignas(4 * sizeof(TA)) Piece { TA x[4]; };
  const int piece = threadIdx.x & (lanes - 1), n_rows = a.n_tokens * a.n_heads;
  const int at = blockIdx.x * (256 / lanes) + threadIdx.x / lanes, row = min(at, n_rows - 1);
  const int t = row / a.n_heads, h = row - t * a.n_heads, c = h * a.dv + piece * 4;
  float4 o = *reinterpret_cast<const float4*>(a.o + (size_t)row * a.dv + piece * 4);
  const Piece gate = *reinterpret_cast<const Piece*>(reinterpret_cast<const TA*>(a.gate) + (size_t)t * a.gate_stride + c);
  float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
  if (a.w) w = *reinterpret_cast<const float4*>(a.w + (a.w_shared ? piece * 4 : c));
  if (a.nq) {
    const float id = 1.0f / (fmaxf(fabsf(a.nq[row]), a.floor_[row]) + a.den_eps);
    o.x *= id; o.y *= id; o.z *= id; o.w *= id;
  }
  float ss = fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, o.w * o.w)));
  for (int off = lanes / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  const float inv = 1.0f / sqrtf(ss / (float)a.dv + a.eps) * a.out_scale;
  auto gated = [&](float v, float weight, TA g) {
    const float x = to_float(g);
    return from_float<TA>(v * inv * weight * (a.silu ? rec_silu(x) : rec_sigmoid(x)));
  };
  Piece y;
  y.x[0] = gated(o.x, w.x, gate.x[0]);
  y.x[1] = gated(o.y, w.y, gate.x[1]);
  y.x[2] = gated(o.z, w.z, gate.x[2]);
  y.x[3] = gated(o.w, w.w, gate.x[3]);
  if (at < n_rows) *reinterpret_cast<Piece*>(reinterpret_cast<TA*>(a.out) + (size_t)t * a.out_stride + c) = y;
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
  const int lanes = a.dv / 4, rows = 256 / lanes;
  const long long n_rows = (long long)a.n_tokens * a.n_heads;
  head_out_kernel<TA><<<(unsigned)((n_rows + rows - 1) / rows), 256, 0, stream>>>(a, lanes);
}
