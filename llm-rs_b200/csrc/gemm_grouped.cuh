// The arguments that the kernels of many small products share (gemm_grouped.cu, gemm_grouped_tc.cu).
#pragma once
#include "common.cuh"

struct GroupedGemmArgs {
  const void* x;            // rows of X
  long long x_stride;       // elements between rows
  long long x_batch;        // elements between batches (batched mode)
  const void* w;            // [groups, N, K]
  const void* w2;           // second weights of the gated unit, or null
  long long w_batch;        // elements between groups
  void* out;
  long long out_stride, out_batch;
  int M, N, K;              // M: rows (batched mode) or total sorted rows (grouped mode)
  const int* tiles;         // grouped mode: [tile][3] = group, first row, rows; null in batched mode
  const int* n_tiles;       // grouped mode: number of tiles on the device
  const int* src;           // grouped mode: sorted row -> row of X (null: the row itself)
  int round_x;
  int tile_rows;            // grouped mode: the most rows a tile of the list has (64 or 128)
  GatedUnit unit;           // EPI_UNIT
  const float* r_bias;      // EPI_GATES: [groups * N] each
  const float* i_bias;
  const float* rate;
};

// gemm_grouped_tc.cu: x_rows rows of X, `groups` weights; `batches` of the batched mode, `max_tiles` of the grouped one.
int launch_grouped_tc(const GroupedGemmArgs& a, int out_dtype, int x_rows, int groups, int batches, int max_tiles,
                      int* error_flag, cudaStream_t stream);
