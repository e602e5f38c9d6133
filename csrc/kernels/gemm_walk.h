// Host interface of the GEMM that walks many tiles per CTA (gemm_walk.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace orinfer {

struct WalkCall {
  const int8_t* a;
  const float* a_scale;
  const void* w;
  const __half* w_scale;
  __half* out;                  // [M, N], columns [0, n_end) are written
  int M, N, K, n_end;
  const int* tiles;             // expert tile table, nullptr: an ordinary product
  const int* meta;
  long long w_stride;           // bytes between experts' banks
  int experts, max_tiles;
};

// Entries that the tile table of a grouped call may have.
int walk_list_room(int fmt);
// mt: 128-row tiles per CTA tile, 1 or 2.
int qgemm_walk_dispatch(int fmt, int mt, const WalkCall& call, cudaStream_t stream);

}  // namespace orinfer
