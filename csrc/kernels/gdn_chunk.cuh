// What the two kernels of long recurrent runs share: the segment table, the sizes of a chunk,
// warp-level tensor-core helpers and exponentials of sums kept in FP64.
#pragma once

#include "common.cuh"

namespace orinfer {

// The state slot of a segment is row_slot[row_start]; a segment whose first row sits at
// position 0 of its request starts from a zero state and a zero history, so a reused slot
// needs no reset.
struct Segment {
  int row_start, rows, pad0, pad1;
};

// Runs of at least this many rows are taken in chunks (see gdn_chunk_kernel).
constexpr int GDN_LONG_ROWS = 40;
constexpr int CHUNK = 32;

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p))
               : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p))
               : "memory");
}
// D += A B on 16 x 8 x 8 TF32 tiles: lane (g, t) holds A rows g, g + 8 at k = t (a0, a1) and
// k = t + 4 (a2, a3), B column g at k = t and t + 4.
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}
// largest value of the four lanes that share a row
__device__ __forceinline__ float quad_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
}
// e with |x| < 2^e (at least -100, at most 129) and powers of two
__device__ __forceinline__ int bound_exp(float x) {
  return max(-100, static_cast<int>((__float_as_uint(x) >> 23) & 255u) - 126);
}
__device__ __forceinline__ float pow2i(int e) {
  return __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
}

// e^x, x FP64: the FP32 exponential of the rounded argument, corrected by what the rounding lost
__device__ __forceinline__ float exp_pair(double x) {
  const float hi = static_cast<float>(x);
  const float e = expf(hi);
  return fmaf(e, static_cast<float>(x - static_cast<double>(hi)), e);
}

// The kernel of gdn_pipe.cu: one CTA per SM, for launches of few or long runs.
int gdn_pipe_launch(const __half* qkv, int conv_dim, const float* ab, const float* a_log,
                    const float* dt_bias, const Segment* segs, int n_segs, const int* row_slot,
                    const int* row_pos, int hk, int hv, float* state, float* out,
                    cudaStream_t stream);

}  // namespace orinfer
