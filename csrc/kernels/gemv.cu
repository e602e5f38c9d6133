// Small-M quantised GEMM (decode path, M <= 8, and up to 16): weight-bandwidth bound.  Each CTA
// owns a few output rows and streams their weights once; lanes decode E8P codes through a
// shared-memory value table and the products with the INT8 activations staged in shared
// memory run on the tensor cores (mma.sync, 16 weight rows x 8 activation rows), or by dp4a for
// small products.  Replaces the reference's dp4a / gemv projections
// (kernels/cuda/model/integer_core.py:275,
// kernels/cuda/model/integer_vq.py:381 integer_e8p_gemv,
// kernels/cuda/model/int8_projection.py:66).
#include "api.h"
#include "common.cuh"
#include "tp_comm.cuh"

namespace orinfer {

constexpr int W8_WARPS = 8;

template <int MT>
__device__ __forceinline__ void stage_activations(int8_t* dst, const int8_t* a, int M, int K) {
  const int chunks = MT * K / 16;
  for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
    const int m = (c * 16) / K;
    int4 v = make_int4(0, 0, 0, 0);
    if (m < M) v = *reinterpret_cast<const int4*>(a + static_cast<size_t>(c) * 16);
    *reinterpret_cast<int4*>(dst + static_cast<size_t>(c) * 16) = v;
  }
}

template <int MT>
__device__ __forceinline__ void store_row(void* out, int out_f32, int m, int n, int N, int acc,
                                          float sw, float sa, const PeerOut* po = nullptr) {
  const float v = (static_cast<float>(acc) * sw) * sa;
  if (po != nullptr) {
    // partial result -> slot [rank] of every rank's inbox (plain peer stores over NVLink)
    const __half hv = __float2half_rn(v);
    const size_t off = (static_cast<size_t>(po->rank) * po->rows_cap + m) * N + n;
    for (int d = 0; d < po->tp; ++d) po->inbox[d][off] = hv;
    return;
  }
  if (out_f32) reinterpret_cast<float*>(out)[static_cast<size_t>(m) * N + n] = v;
  else reinterpret_cast<__half*>(out)[static_cast<size_t>(m) * N + n] = __float2half_rn(v);
}

// FMT 0: INT8 weights, 1: Q4 (U32 codes), 2: Q2 (U16 codes).  One persistent CTA per SM: the
// decode tables (32 interleaved copies, so a lane's lookups never meet another lane's on a
// bank, and an address is one byte permute: see E8pRows) and the activations are staged once.  The
// grid is n_parts x k_parts CTAs; a CTA owns a contiguous range of 16-row groups and one range of
// 128-wide k-blocks, its warps take contiguous runs of (group, k-block) units, every lane keeps
// DEPTH units of weight loads in flight (the first ones are issued before the tables are filled,
// except in the fused forms), and the partial dot products meet in shared memory (integer atomics:
// exact, so the result does not depend on the order).
//
// Products: m16n8k32 INT8 MMAs with the weights as A (lane (g, t) holds rows g and g + 8) and
// the activation rows as the eight columns of B.  A lane's four code words of a k-block are
// weight octets 4t .. 4t + 3; step j multiplies octets {4t + j}, so the activations are staged
// octet-wise as [k-block][j][t][row] and a step reads 8 bytes per lane without a bank conflict.
// One MMA replaces 4 M dp4a and 2 M shared-memory loads: the time no longer grows with M.
//
// 8 x 19456 x 2560 18.0 -> 16.3 us, 8 x 2560 x 4096 9.9 -> 8.9, 4 x 6144 x 2560 9.6 -> 8.6 with the
// permuted addresses and the small loads ahead of the weights (see GemvEarly).
//
// The decode never forms the weights.  With v the 4-bit fields of a code (common.cuh), a Q4
// weight is 8*v0 + 2*v1 - 75, so
//     sum_k a_k w_k = 2 * sum_k a_k (4*v0 + v1)_k  -  75 * sum_k a_k
// and the first sum multiplies bytes built with two masks and one multiply-add; sum_k a_k is
// computed once per activation row while it is staged.  Q2 likewise with 2*v - 15.
//
// k_parts > 1 (E8P projections too narrow for one CTA per SM): the CTAs of one n-part add their
// integers into a zeroed workspace; the last one to finish (ticket) applies the scales,
// writes the outputs and zeroes what it read.  Launches that use the workspace must not
// overlap on the device (they are issued on one stream).
constexpr int GEMV_THREADS = 1024;
constexpr size_t GEMV_SMEM_LIMIT = 220 * 1024;

__device__ __forceinline__ void mma_i8_16832(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                             uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Weights of one (group, k-block) unit as loaded by a lane: rows g and g + 8.
template <int FMT>
struct GemvUnit {
  static constexpr int WORDS = FMT == 0 ? 8 : (FMT == 1 ? 4 : 2);    // 32-bit words per row
  uint32_t w[2][WORDS];
};

// Position of channel k of activation row m in the staged activations (bytes).  dp4a: rows as they
// are (a warp reads four octets 32 bytes apart); E8P MMAs: octets ordered
// [k-block][octet % 4][octet / 4][row]; INT8 weights: 16-byte pieces ordered
// [64 channels][row][piece], a lane's pieces being two steps each.
template <int FMT, int MT, bool DP4A>
__device__ __forceinline__ int act_pos(int m, int k, int K) {
  if (DP4A) return m * K + k;
  if (MT == 16)                                  // two planes of eight rows, as the MMAs take them
    return (m >> 3) * 8 * K + act_pos<FMT, MT == 16 ? 8 : MT, false>(m & 7, k, K);
  if (FMT == 0) return ((k >> 6) * MT + m) * 64 + (k & 63);
  const int o = (k >> 3) & 15;
  return (((k >> 7) * 16 + (o & 3) * 4 + (o >> 2)) * MT + m) * 8 + (k & 7);
}

// Optional fusion of the decode step's row kernels into the projection (at most 8 rows, no
// peers).  `pre` builds the INT8 activations inside every CTA instead of reading them:
//   1: rows = resid (+ x), RMSNorm with norm_w, rotation, A8        (x and norm_w may be null)
//   2: rows = x (FP16 [M, K]), rotation, A8
//   3: rows = SwiGLU of x (FP16 [M, 2K]: gate | up), rotation, A8
// with exactly the arithmetic of act_prep_kernel (same helpers, same order), so a row gives
// the same bits through either path.  Every CTA repeats the (small) row preparation; CTA 0
// also stores what other kernels may read (y_out, q_out, scale_out).  `resid_accum` adds the
// FP16-rounded output into an FP32 matrix: the residual stream then already contains the
// branch output when the next prologue reads it, so no kernel both reads and writes it.
struct GemvFuse {
  int pre;
  const __half* x;
  const float* resid;
  const __half* norm_w;
  const int8_t* signs;
  float eps;
  int zero_centered;
  int8_t* q_out;
  float* scale_out;
  __half* y_out;
  float* resid_accum;
};

// What a CTA needs before its first product besides weights: the decode tables, the activation rows
// and the scales.  They are requested ahead of the weights.  Behind them they waited for a CTA's
// first 64 KB, three times in a row: the first product came 5 us into the 13 us of 1 x 19456 x
// 2560, 6 us into the 8 us of 8 x 2560 x 4096.
template <int FMT, int THREADS>
struct GemvEarly {
  static constexpr int ROWS = 2;                 // 16-byte pieces of the rows per thread
  E8pFill<THREADS> fill;
  int4 rows[ROWS];
  float scale;
  __half w_scale;
  __device__ __forceinline__ void load(const E8pTables* __restrict__ tables,
                                       const int8_t* a, const float* a_scale, const __half* ws,
                                       int n_count, int M, int K, bool plain, int tid) {
    if (FMT != 0) fill.load(tables, tid);
    grid_wait();
    grid_release();
    w_scale = tid < n_count ? ws[tid] : __half(0.f);
    scale = 0.f;
    if (plain) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int c = tid + i * THREADS;
        rows[i] = c * 16 < M * K ? reinterpret_cast<const int4*>(a)[c]
                                 : make_int4(0, 0, 0, 0);
      }
      if (tid < M) scale = a_scale[tid];
    }
  }
  // the tables, the outputs' scales (sw) and zeroed sums
  __device__ __forceinline__ void store(unsigned char* smem, float* sw,
                                        const __half* ws, int n_count, int* sums, int n_sums,
                                        int tid) const {
    if (FMT != 0) fill.store(smem, tid);
    if (tid < n_count) sw[tid] = __half2float(w_scale);
    for (int i = tid + THREADS; i < n_count; i += THREADS) sw[i] = __half2float(ws[i]);
    for (int i = tid; i < n_sums; i += THREADS) sums[i] = 0;
  }
};

// Fills the staged activations, their row sums (asum, zeroed before) and their scales: from INT8
// rows, or by the row preparation of fz.pre, one row at a time in fbuf [K].
template <int FMT, int MT, int THREADS, bool DP4A>
__device__ __forceinline__ void gemv_rows(int8_t* act, int* asum, float* scale_s, float* fbuf,
                                          float* red, float* blk_sum, const int8_t* a,
                                          const float* a_scale, int M, int K,
                                          const GemvFuse& fz,
                                          const GemvEarly<FMT, THREADS>& early) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (FMT == 0 || fz.pre == 0) {
    // stage the activations; their row sums ride along
    const int chunks = MT * K / 16;
    int part_sum[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) part_sum[m] = 0;
    auto place = [&](int c, const int4& v) {
      const int m = (c * 16) / K, k = c * 16 - m * K;
      *reinterpret_cast<int2*>(act + act_pos<FMT, MT, DP4A>(m, k, K)) = make_int2(v.x, v.y);
      *reinterpret_cast<int2*>(act + act_pos<FMT, MT, DP4A>(m, k + 8, K)) = make_int2(v.z, v.w);
      int s = __dp4a(v.x, 0x01010101, 0);
      s = __dp4a(v.y, 0x01010101, s);
      s = __dp4a(v.z, 0x01010101, s);
      s = __dp4a(v.w, 0x01010101, s);
#pragma unroll
      for (int mm = 0; mm < MT; ++mm)
        if (mm == m) part_sum[mm] += s;
    };
#pragma unroll
    for (int i = 0; i < early.ROWS; ++i)
      if (tid + i * THREADS < chunks) place(tid + i * THREADS, early.rows[i]);
    for (int c = tid + early.ROWS * THREADS; c < chunks; c += THREADS) {
      int4 v = make_int4(0, 0, 0, 0);
      if (c * 16 < M * K) v = *reinterpret_cast<const int4*>(a + static_cast<size_t>(c) * 16);
      place(c, v);
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      int s = part_sum[m];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0 && s != 0) atomicAdd(&asum[m], s);
    }
    if (tid < MT) scale_s[tid] = early.scale;
  } else {
    // build the activations: the row kernels' work, repeated by every CTA
    constexpr int NWP = THREADS / 32;
    const bool first_cta = blockIdx.x == 0;
    for (int m = 0; m < MT; ++m) {
      if (m >= M) break;                         // columns past the last row are not used
      float* fb = fbuf;                          // one row at a time
      if (fz.pre == 3) {
        const __half* g = fz.x + static_cast<size_t>(m) * 2 * K;
        const __half* u = g + K;
        for (int i = tid * 8; i < K; i += THREADS * 8) {
          const int4 gr = *reinterpret_cast<const int4*>(g + i);
          const int4 ur = *reinterpret_cast<const int4*>(u + i);
          const __half* gh = reinterpret_cast<const __half*>(&gr);
          const __half* uh = reinterpret_cast<const __half*>(&ur);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float gv = __half2float(gh[j]);
            const float sg = sigmoid_f32(gv);
            fb[i + j] = round_f16(__fmul_rn(__fmul_rn(gv, sg), __half2float(uh[j])));
          }
        }
      } else {
        const __half* xr = fz.x ? fz.x + static_cast<size_t>(m) * K : nullptr;
        const float* rr = (fz.pre == 1 && fz.resid) ? fz.resid + static_cast<size_t>(m) * K
                                                    : nullptr;
        for (int i = tid * 8; i < K; i += THREADS * 8) {
          float v[8];
          if (xr) {
            const int4 raw = *reinterpret_cast<const int4*>(xr + i);
            const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __half2float(h[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = 0.f;
          }
          if (rr) {
            const float4 r0 = *reinterpret_cast<const float4*>(rr + i);
            const float4 r1 = *reinterpret_cast<const float4*>(rr + i + 4);
            v[0] += r0.x; v[1] += r0.y; v[2] += r0.z; v[3] += r0.w;
            v[4] += r1.x; v[5] += r1.y; v[6] += r1.z; v[7] += r1.w;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) fb[i + j] = v[j];
        }
        if (fz.norm_w) {
          __syncthreads();
          for (int b = warp; b < K / 128; b += NWP) {
            const float sq = block128_sumsq(fb + b * 128, lane);
            if (lane == 0) blk_sum[b] = sq;
          }
          __syncthreads();
          float total = 0.f;
          for (int b = 0; b < K / 128; ++b) total = __fadd_rn(total, blk_sum[b]);
          const float r = rsqrtf(total / static_cast<float>(K) + fz.eps);
          const float add = fz.zero_centered ? 1.f : 0.f;
          for (int i = tid * 8; i < K; i += THREADS * 8) {
            const int4 wr = *reinterpret_cast<const int4*>(fz.norm_w + i);
            const __half* wh = reinterpret_cast<const __half*>(&wr);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              fb[i + j] = round_f16(__fmul_rn(__fmul_rn(fb[i + j], r), __half2float(wh[j]) + add));
          }
        } else {
          for (int i = tid * 8; i < K; i += THREADS * 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) fb[i + j] = round_f16(fb[i + j]);
        }
      }
      __syncthreads();
      if (fz.y_out != nullptr && first_cta) {
        __half* yr = fz.y_out + static_cast<size_t>(m) * K;
        for (int i = tid * 8; i < K; i += THREADS * 8) {
          __align__(16) __half h[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) h[j] = __float2half_rn(fb[i + j]);
          *reinterpret_cast<int4*>(yr + i) = *reinterpret_cast<const int4*>(h);
        }
      }
      float amax = 0.f;
      if (fz.signs) {
        for (int b = warp; b < K / 128; b += NWP)
          amax = fmaxf(amax, hadamard128_inplace(fb + b * 128, fz.signs + b * 128, lane));
      } else {
        for (int i = tid; i < K; i += THREADS) amax = fmaxf(amax, fabsf(fb[i]));
      }
      amax = block_reduce(amax, red, true);
      const float scale = a8_scale(amax);
      int psum = 0;
      for (int i = tid * 4; i < K; i += THREADS * 4) {
        char4 c;
        c.x = static_cast<signed char>(a8_code(fb[i + 0], scale));
        c.y = static_cast<signed char>(a8_code(fb[i + 1], scale));
        c.z = static_cast<signed char>(a8_code(fb[i + 2], scale));
        c.w = static_cast<signed char>(a8_code(fb[i + 3], scale));
        *reinterpret_cast<char4*>(act + act_pos<FMT, MT, DP4A>(m, i, K)) = c;
        if (fz.q_out != nullptr && first_cta)
          *reinterpret_cast<char4*>(fz.q_out + static_cast<size_t>(m) * K + i) = c;
        psum = __dp4a(*reinterpret_cast<const int*>(&c), 0x01010101, psum);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
      if (lane == 0 && psum != 0) atomicAdd(&asum[m], psum);
      if (tid == 0) {
        scale_s[m] = scale;
        if (fz.scale_out != nullptr && first_cta) fz.scale_out[m] = scale;
      }
      __syncthreads();
    }
  }
}

// Scales and writes the outputs n_base .. n_base + n_count from the integers in acc_s.
template <int FMT, int MT, int THREADS>
__device__ __forceinline__ void gemv_finish(int* acc_s, const int* asum, const float* scale_s,
                                            int* last_flag, const float* sw_s,
                                            void* __restrict__ out, int M, int N, int out_f32,
                                            const PeerOut& po, int ll_seq, int np, int k_parts,
                                            int n_base, int n_count, int* ws,
                                            const GemvFuse& fz) {
  const int tid = threadIdx.x;
  const PeerOut* peer = po.tp > 0 ? &po : nullptr;
  const bool ll = peer != nullptr && po.rows_per == LL_MODE;
  // sum_k a_k w_k from the staged integers: Q4 2*acc - 75*S, Q2 2*acc - 15*S
  constexpr int UNIT = FMT == 0 ? 1 : 2, BIAS = FMT == 0 ? 0 : (FMT == 1 ? 75 : 15);
  constexpr size_t WS_COLS = MT > 8 ? GEMV_WS_COLS / 2 : GEMV_WS_COLS;
  bool finalize = true;
  if (k_parts > 1) {
    // add this CTA's integers to the workspace; the last CTA of the n-part finishes
    for (int i = tid; i < n_count * MT; i += THREADS) {
      const int m = i / n_count, r = i % n_count;
      const int v = acc_s[r * MT + m];
      if (m < M && v != 0) atomicAdd(ws + m * WS_COLS + n_base + r, v);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      unsigned int* ticket = reinterpret_cast<unsigned int*>(ws + 8 * GEMV_WS_COLS) + np;
      const unsigned int t = atomicAdd(ticket, 1u);
      *last_flag = t == static_cast<unsigned int>(k_parts - 1);
      if (*last_flag) *ticket = 0;
    }
    __syncthreads();
    finalize = *last_flag != 0;
    if (finalize) {
      __threadfence();
      for (int i = tid; i < n_count * MT; i += THREADS) {
        const int m = i / n_count, r = i % n_count;
        int v = 0;
        if (m < M) {
          int* p = ws + m * WS_COLS + n_base + r;
          v = __ldcg(p);
          *p = 0;
        }
        acc_s[r * MT + m] = v;
      }
      __syncthreads();
    }
  }
  if (finalize) {
    if (peer != nullptr && n_count % 8 == 0) {
      // peers get whole 16-byte segments (8 consecutive outputs of one row per store):
      // 2-byte remote stores would each become their own NVLink write
      const int segs = n_count / 8;
      for (int i = tid; i < segs * MT; i += THREADS) {
        const int m = i / segs, seg = i % segs;
        if (m < M) {
          __align__(16) __half h[8];
          const float sa = scale_s[m];
          const int bias = BIAS * asum[m];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const int total = UNIT * acc_s[(seg * 8 + r) * MT + m] - bias;
            h[r] = __float2half_rn(
                (static_cast<float>(total) * sw_s[seg * 8 + r]) * sa);
          }
          if (ll) {
            ll_store8(po, ll_seq, m, n_base + seg * 8, N, h);
          } else {
            const size_t off =
                (static_cast<size_t>(po.rank) * po.rows_cap + m) * N + n_base + seg * 8;
            for (int d = 0; d < po.tp; ++d)
              *reinterpret_cast<int4*>(po.inbox[d] + off) = *reinterpret_cast<const int4*>(h);
          }
        }
      }
    } else {
      for (int i = tid; i < n_count * MT; i += THREADS) {
        const int m = i / n_count, r = i % n_count;
        if (m < M) {
          const int total = UNIT * acc_s[r * MT + m] - BIAS * asum[m];
          const float sw = sw_s[r];
          if (FMT != 0 && fz.resid_accum != nullptr) {
            const __half hv = __float2half_rn((static_cast<float>(total) * sw) * scale_s[m]);
            float* dst = fz.resid_accum + static_cast<size_t>(m) * N + n_base + r;
            *dst = *dst + __half2float(hv);
            if (out != nullptr)
              reinterpret_cast<__half*>(out)[static_cast<size_t>(m) * N + n_base + r] = hv;
          } else {
            store_row<MT>(out, out_f32, m, n_base + r, N, total, sw, scale_s[m], peer);
          }
        }
      }
    }
  }
  if (ll) ll_done(po, ll_seq, gridDim.x);
  else if (peer != nullptr) peer_signal_done(po, gridDim.x);
}

template <int FMT, int MT>
__global__ void __launch_bounds__(GEMV_THREADS, 1) qgemv_kernel(
    const int8_t* a, const float* a_scale, const void* w, const __half* w_scale,
    void* __restrict__ out, int M, int N, int K, int out_f32, const E8pTables* __restrict__ tables,
    PeerOut po, int n_parts, int k_parts, int max_groups, int* ws, GemvFuse fz) {
  constexpr int THREADS = GEMV_THREADS;
  constexpr int ROWS = 16, DEPTH = FMT == 2 ? 4 : 2;     // rows of a group, units in flight
  using Unit = GemvUnit<FMT>;
  constexpr int LUT_BYTES = FMT == 0 ? 0 : static_cast<int>(sizeof(E8pRows));
  const bool ll = po.tp > 0 && po.rows_per == LL_MODE;
  const int ll_seq = ll ? *reinterpret_cast<volatile int*>(po.sent) + 1 : 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int8_t* act = reinterpret_cast<int8_t*>(smem_raw) + LUT_BYTES;
  int* acc_s = reinterpret_cast<int*>(act + static_cast<size_t>(MT) * K);   // [16 max_groups][MT]
  int* asum = acc_s + max_groups * 16 * MT;                                  // [MT]
  float* scale_s = reinterpret_cast<float*>(asum + MT);                      // [MT]
  float* sw_s = scale_s + MT;                                                // [16 max_groups]
  float* fbuf = reinterpret_cast<float*>(                                    // [K], pre only
      (reinterpret_cast<uintptr_t>(sw_s + max_groups * 16) + 15) & ~static_cast<uintptr_t>(15));
  __shared__ int last_flag;
  __shared__ float red[32];
  __shared__ float blk_sum[128];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int kb_all = K / 128;
  // a CTA's rows are a multiple of eight (the SMs then differ by 8 rows, not 16); its last group
  // may be half a group
  const int oct = N / 8;
  const int np = blockIdx.x % n_parts, kp = blockIdx.x / n_parts;
  const int n_base = static_cast<int>(static_cast<long long>(oct) * np / n_parts) * 8;
  const int n_count =
      static_cast<int>(static_cast<long long>(oct) * (np + 1) / n_parts) * 8 - n_base;
  const int groups = (n_count + ROWS - 1) / ROWS;
  const int kb_lo = kb_all * kp / k_parts, kb_hi = kb_all * (kp + 1) / k_parts;
  const int kbs = kb_hi - kb_lo;
  const int units = groups * kbs;
  constexpr int NW = THREADS / 32;
  const int u_lo = static_cast<int>(static_cast<long long>(units) * warp / NW);
  const int u_hi = static_cast<int>(static_cast<long long>(units) * (warp + 1) / NW);
  // (group, k-block) of the unit being loaded, and of the unit being consumed
  int lg = 0, lkb = 0;
  if (u_lo < u_hi) {
    lg = u_lo / kbs;
    lkb = kb_lo + u_lo % kbs;
  }
  int cg = lg, ckb = lkb;
  Unit buf[DEPTH];
  auto fetch = [&](Unit& v, int uu) {
    if (uu >= u_hi) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && lg * ROWS + 8 >= n_count) break;       // half a group
      const int n = n_base + lg * ROWS + g + h * 8;
      if (FMT == 0) {
        const uint4* p = reinterpret_cast<const uint4*>(w) + static_cast<size_t>(n) * (K / 16) +
                         lkb * 8 + t;
        const uint4 x = *p, y = p[4];
        v.w[h][0] = x.x; v.w[h][1] = x.y; v.w[h][2] = x.z; v.w[h][3] = x.w;
        v.w[h][4 % Unit::WORDS] = y.x; v.w[h][5 % Unit::WORDS] = y.y;
        v.w[h][6 % Unit::WORDS] = y.z; v.w[h][7 % Unit::WORDS] = y.w;
      } else if (FMT == 1) {
        const uint4 x =
            reinterpret_cast<const uint4*>(w)[(static_cast<size_t>(lkb) * N + n) * 4 + t];
        v.w[h][0] = x.x; v.w[h][1] = x.y;
        v.w[h][2 % Unit::WORDS] = x.z; v.w[h][3 % Unit::WORDS] = x.w;
      } else {
        const uint2 x =
            reinterpret_cast<const uint2*>(w)[(static_cast<size_t>(lkb) * N + n) * 4 + t];
        v.w[h][0] = x.x; v.w[h][1] = x.y;
      }
    }
    if (++lkb == kb_hi) {
      lkb = kb_lo;
      ++lg;
    }
  };
  // The first weights are requested before the tables are filled, except where the row
  // preparation needs the registers.
  GemvEarly<FMT, THREADS> early;
  early.load(tables, a, a_scale, w_scale + n_base, n_count, M, K, FMT == 0 || fz.pre == 0, tid);
  if (FMT == 0 || fz.pre == 0) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) fetch(buf[i], u_lo + i);
  }
  early.store(smem_raw, sw_s, w_scale + n_base, n_count, acc_s, max_groups * 16 * MT + MT, tid);
  __syncthreads();
  gemv_rows<FMT, MT, THREADS, false>(act, asum, scale_s, fbuf, red, blk_sum, a, a_scale, M, K, fz,
                                     early);
  __syncthreads();

  if (FMT != 0 && fz.pre != 0) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) fetch(buf[i], u_lo + i);
  }
  constexpr int COLS = MT == 16 ? 2 : 1;           // eight activation rows each
  constexpr int MC = MT == 16 ? 8 : MT;
  int acc[COLS][4] = {};
  const uint32_t lane4 = lane * 4;
  for (int base = u_lo; base < u_hi; base += DEPTH) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) {
      if (base + i < u_hi) {
        const bool half = cg * ROWS + 8 >= n_count;
        if (FMT == 0) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            int4 b[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
              b[c] = make_int4(0, 0, 0, 0);
              if (g < MC)
                b[c] = *reinterpret_cast<const int4*>(
                    act + act_pos<FMT, MT, false>(g + 8 * c, ckb * 128 + j * 64 + t * 16, K));
            }
            const uint32_t* r0 = buf[i].w[0] + (j * 4) % Unit::WORDS;
            const uint32_t* r1 = buf[i].w[1] + (j * 4) % Unit::WORDS;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
              mma_i8_16832(acc[c], r0[0], r1[0], r0[1], r1[1], b[c].x, b[c].y);
              mma_i8_16832(acc[c], r0[2 % Unit::WORDS], r1[2 % Unit::WORDS], r0[3 % Unit::WORDS],
                           r1[3 % Unit::WORDS], b[c].z, b[c].w);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            int2 b[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
              b[c] = make_int2(0, 0);
              if (g < MC)
                b[c] = *reinterpret_cast<const int2*>(
                    act + c * 8 * K + ((ckb * 16 + j * 4 + t) * MC + g) * 8);
            }
            uint32_t lo[2] = {0u, 0u}, hi[2] = {0u, 0u};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (h == 1 && half) break;
              const uint32_t word = buf[i].w[h][(FMT == 1 ? j : j >> 1) % Unit::WORDS];
              const uint2 v = FMT == 1 ? e8p_bytes_q4(word, smem_raw, lane4)
                              : j & 1  ? e8p_bytes_q2<1>(word, smem_raw, lane4)
                                       : e8p_bytes_q2<0>(word, smem_raw, lane4);
              lo[h] = v.x;
              hi[h] = v.y;
            }
#pragma unroll
            for (int c = 0; c < COLS; ++c)
              mma_i8_16832(acc[c], lo[0], lo[1], hi[0], hi[1], b[c].x, b[c].y);
          }
        }
        fetch(buf[i], base + i + DEPTH);
        const bool last_of_group = ckb + 1 == kb_hi, last_unit = base + i + 1 == u_hi;
        if (last_of_group || last_unit) {
#pragma unroll
          for (int c = 0; c < COLS; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int m = 2 * t + (e & 1) + 8 * c;
              if (m < MT && !(half && e >= 2))
                atomicAdd(&acc_s[(cg * ROWS + g + (e >> 1) * 8) * MT + m], acc[c][e]);
              acc[c][e] = 0;
            }
        }
        if (last_of_group) {
          ckb = kb_lo;
          ++cg;
        } else {
          ++ckb;
        }
      }
    }
  }
  __syncthreads();

  gemv_finish<FMT, MT, THREADS>(acc_s, asum, scale_s, &last_flag, sw_s, out, M, N, out_f32, po,
                                ll_seq, np, k_parts, n_base, n_count, ws, fz);
}

// E8P products by dp4a instead of MMAs (see gemv_dp4a for where).  An MMA spends eight columns on
// however few rows, its form keeps two weight rows and less of them in flight per lane, and its
// registers leave the row preparation little; this one spends two to four dp4a and a read of
// activations per row and code word.  Lane l holds row l / LPR of a group and an LPR-th of the
// k-block, DEPTH units in flight.  1 x 19456 x 2560 14.8 -> 12.9 us, 1 x 2560 x 9728 12.1 -> 10.9,
// 1 x 6144 x 2560 Q2 6.8 -> 6.6 with the fields multiplied as they are looked up and the small
// loads ahead of the weights; with the early start too, eight weights in turn in a graph, one row
// 15.1 -> 11.8, 11.3 -> 9.2 and 6.7 -> 5.7, two rows 16.4 -> 13.9, 12.9 -> 11.0 and 7.5 -> 6.4 (12
// bytes of spills a thread).  About 2 us are launch, 2.5 the first loads, 6 the products (63 % of
// the issue slots, half of the ALU pipe), 1 the outputs.
template <int FMT, int MT>
struct Dp4a {
  static constexpr int THREADS = MT <= 2 ? 1024 : 512;             // registers
};

template <int FMT, int MT>
__global__ void __launch_bounds__(Dp4a<FMT, MT>::THREADS, 1) e8p_dp4a_kernel(
    const int8_t* a, const float* a_scale, const uint4* w, const __half* w_scale,
    void* __restrict__ out, int M, int N, int K, int out_f32, const E8pTables* __restrict__ tables,
    PeerOut po, int n_parts, int k_parts, int max_groups, int* ws, GemvFuse fz) {
  constexpr int THREADS = Dp4a<FMT, MT>::THREADS, DEPTH = 4;
  constexpr int ROWS = FMT == 1 ? 8 : 16;        // output rows of a group
  constexpr int LPR = 32 / ROWS;                 // lanes per row, 16 bytes of codes each
  const bool ll = po.tp > 0 && po.rows_per == LL_MODE;
  const int ll_seq = ll ? *reinterpret_cast<volatile int*>(po.sent) + 1 : 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int8_t* act = reinterpret_cast<int8_t*>(smem_raw) + sizeof(E8pRows);
  int* acc_s = reinterpret_cast<int*>(act + static_cast<size_t>(MT) * K);   // [16 max_groups][MT]
  int* asum = acc_s + max_groups * 16 * MT;                                  // [MT]
  float* scale_s = reinterpret_cast<float*>(asum + MT);                      // [MT]
  float* sw_s = scale_s + MT;                                                // [16 max_groups]
  float* fbuf = reinterpret_cast<float*>(                                    // [K], pre only
      (reinterpret_cast<uintptr_t>(sw_s + max_groups * 16) + 15) & ~static_cast<uintptr_t>(15));
  __shared__ int last_flag;
  __shared__ float red[32];
  __shared__ float blk_sum[128];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = lane / LPR, part = lane % LPR;
  const int kb_all = K / 128, groups = (N + ROWS - 1) / ROWS;
  const int np = blockIdx.x % n_parts, kp = blockIdx.x / n_parts;
  const int g_lo = static_cast<int>(static_cast<long long>(groups) * np / n_parts);
  const int g_hi = static_cast<int>(static_cast<long long>(groups) * (np + 1) / n_parts);
  const int kb_lo = kb_all * kp / k_parts, kb_hi = kb_all * (kp + 1) / k_parts;
  const int kbs = kb_hi - kb_lo;
  const int units = (g_hi - g_lo) * kbs;
  constexpr int NW = THREADS / 32;
  const int u_lo = static_cast<int>(static_cast<long long>(units) * warp / NW);
  const int u_hi = static_cast<int>(static_cast<long long>(units) * (warp + 1) / NW);
  // (group, k-block) of the unit being loaded, and of the unit being consumed
  int lg = g_lo, lkb = kb_lo;
  if (u_lo < u_hi) {
    lg += u_lo / kbs;
    lkb += u_lo % kbs;
  }
  int g = lg, kb = lkb;
  uint4 buf[DEPTH];
  auto fetch = [&](int uu) -> uint4 {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (uu < u_hi) {
      const int n = min(lg * ROWS + row, N - 1);
      v = w[(static_cast<size_t>(lkb) * N + n) * LPR + part];
      if (++lkb == kb_hi) {
        lkb = kb_lo;
        ++lg;
      }
    }
    return v;
  };
  // requested before the tables are filled, except where the row preparation needs the registers
  const int n_base = g_lo * ROWS, n_count = min(g_hi * ROWS, N) - n_base;
  GemvEarly<FMT, THREADS> early;
  early.load(tables, a, a_scale, w_scale + n_base, n_count, M, K, fz.pre == 0, tid);
  if (fz.pre == 0) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) buf[i] = fetch(u_lo + i);
  }
  early.store(smem_raw, sw_s, w_scale + n_base, n_count, acc_s, max_groups * 16 * MT + MT, tid);
  __syncthreads();
  gemv_rows<FMT, MT, THREADS, true>(act, asum, scale_s, fbuf, red, blk_sum, a, a_scale, M, K, fz,
                                    early);
  __syncthreads();
  if (fz.pre != 0) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) buf[i] = fetch(u_lo + i);
  }

  // One or two rows: the fields are multiplied as they come out of the lookup (four dp4a per row
  // and word), the odd ones sixteenfold in sums of their own; more rows: four dp4a would cost more
  // than forming 4 * v0 + v1.
  constexpr bool RAW = FMT == 1 && MT <= 2;
  constexpr int SUMS = RAW ? 4 : 1;
  int acc[MT][SUMS];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int q = 0; q < SUMS; ++q) acc[m][q] = 0;
  const uint32_t lane4 = lane * 4;
  for (int base = u_lo; base < u_hi; base += DEPTH) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) {
      const uint4 cur = buf[i];
      buf[i] = fetch(base + i + DEPTH);
      if (base + i < u_hi) {
        const int8_t* abase = act + kb * 128 + part * (128 / LPR);
        const uint32_t words[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
        for (int j = 0; j < (FMT == 1 ? 4 : 8); ++j) {
          if constexpr (RAW) {
            uint32_t l0, h0, l1, h1;
            e8p_lookup<0>(words[j & 3], smem_raw, lane4, l0, h0);
            e8p_lookup<1>(words[j & 3], smem_raw, lane4, l1, h1);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              const int2 av = *reinterpret_cast<const int2*>(abase + m * K + j * 8);
              acc[m][0] = dp4a_us(l0, av.x, acc[m][0]);
              acc[m][1] = dp4a_us(h0, av.y, acc[m][1]);
              acc[m][2 % SUMS] = dp4a_us(l1, av.x, acc[m][2 % SUMS]);
              acc[m][3 % SUMS] = dp4a_us(h1, av.y, acc[m][3 % SUMS]);
            }
          } else {
            const uint2 v = FMT == 1 ? e8p_bytes_q4(words[j & 3], smem_raw, lane4)
                            : j & 1  ? e8p_bytes_q2<1>(words[j >> 1], smem_raw, lane4)
                                     : e8p_bytes_q2<0>(words[j >> 1], smem_raw, lane4);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              const int2 av = *reinterpret_cast<const int2*>(abase + m * K + j * 8);
              acc[m][0] = dp4a_us(v.x, av.x, acc[m][0]);
              acc[m][0] = dp4a_us(v.y, av.y, acc[m][0]);
            }
          }
        }
        const bool last_of_group = kb + 1 == kb_hi, last_unit = base + i + 1 == u_hi;
        if (last_of_group || last_unit) {
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            int v = acc[m][0];
            if (RAW)
              v = 4 * (v + acc[m][1 % SUMS] / 16) + acc[m][2 % SUMS] + acc[m][3 % SUMS] / 16;
#pragma unroll
            for (int o = 1; o < LPR; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (part == 0) atomicAdd(&acc_s[((g - g_lo) * ROWS + row) * MT + m], v);
#pragma unroll
            for (int q = 0; q < SUMS; ++q) acc[m][q] = 0;
          }
        }
        if (last_of_group) {
          kb = kb_lo;
          ++g;
        } else {
          ++kb;
        }
      }
    }
  }
  __syncthreads();
  gemv_finish<FMT, MT, THREADS>(acc_s, asum, scale_s, &last_flag, sw_s, out, M, N, out_f32, po,
                                ll_seq, np, k_parts, n_base, n_count, ws, fz);
}

// INT8 weights by one warp per output row: 16 weights per lane per step, as many CTAs as rows
// need, the activations read from shared memory once per weight row.  Small projections are up to
// twice as fast this way as with the persistent CTAs of the MMA form; from three rows on its reads
// lose to the MMAs once there is work for every SM.
//   one row: 6144 x 2560 3.7 us against 6.9, a 151936-row head 74 against 75 (with peers: on one
//     GPU such a head is a stream, see w8_streams)
//   four: 1024 x 1024 2.7 against 5.2, 4096 x 4096 6.0 against 6.9, 5120 x 9728 15.7 against 16.2,
//     6144 x 2560 7.4 against 6.7, 9728 x 1024 5.8 against 6.0, 12288 x 1024 7.0 against 6.1
//   eight: 1024 x 1024 4.0 against 5.9, 2048 x 4096 6.5 against 6.9, 4096 x 2560 7.7 against 7.2,
//     512 x 9728 9.4 against 8.8, head 205 against 77
inline bool w8_by_rows(int M, int N, int K) {
  const long long cells = static_cast<long long>(N) * K;
  if (M <= 2) return true;
  if (M <= 4) return K <= 16384 && (N < 6144 || (N < 12288 && cells < 12500000));
  return K <= 8192 && cells <= 8 * 1024 * 1024;
}

template <int MT>
__global__ void __launch_bounds__(W8_WARPS * 32) w8_gemv_kernel(
    const int8_t* a, const float* a_scale, const int8_t* w, const __half* w_scale,
    void* __restrict__ out, int M, int N, int K, int out_f32, PeerOut po) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_wait();
  grid_release();
  int8_t* act = reinterpret_cast<int8_t*>(smem_raw);
  const PeerOut* peer = po.tp > 0 ? &po : nullptr;
  stage_activations<MT>(act, a, M, K);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * W8_WARPS + warp;
  if (n < N) {
  const int8_t* wr = w + static_cast<size_t>(n) * K;
  int acc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = 0;
#pragma unroll 4
  for (int k = lane * 16; k < K; k += 512) {
    const int4 wv = *reinterpret_cast<const int4*>(wr + k);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int4 av = *reinterpret_cast<const int4*>(act + m * K + k);
      acc[m] = __dp4a(wv.x, av.x, acc[m]);
      acc[m] = __dp4a(wv.y, av.y, acc[m]);
      acc[m] = __dp4a(wv.z, av.z, acc[m]);
      acc[m] = __dp4a(wv.w, av.w, acc[m]);
    }
  }
  const float sw = __half2float(w_scale[n]);
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    int v = acc[m];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0 && m < M) store_row<MT>(out, out_f32, m, n, N, v, sw, a_scale[m], peer);
  }
  }
  if (peer != nullptr) peer_signal_done(po, gridDim.x);
}

// Large INT8 projections (the vocabulary head): a stream.  The forms above walk many short pieces
// of rows at once (16 rows x 128 bytes per warp, or one row per warp), which left DRAM at 5 TB/s
// however many loads were in flight.  Here a CTA per SM takes tiles of 16 whole rows, neighbouring
// CTAs neighbouring tiles, so that all of them read one region of the matrix; a warp copies rows
// into a ring with bulk copies, and each stage of the ring has a warp of its own that multiplies
// the tile it holds (MMAs as above: 16 weight rows x 8 activation rows) and stores its outputs.
// Rows lie 64 bytes past a multiple of 128 apart in shared memory, so 16-byte reads of two rows
// meet on no bank. 151936 x 2560 (389 MB): one row 75 -> 57.6 us (6.75 TB/s, with four matrices in
// turn as with one: reads alone, above the 6.54 TB/s of a copy), two 79 -> 58.4, four 76 -> 60.2,
// eight 78 -> 63.7.  Below about 24 M weights the set-up of the rings costs more than it gives:
// one row of 12288 x 2560 9.3 -> 9.1 us, eight rows 12.5 both ways, but 6144 x 2560 5.7 -> 6.7 and
// 9.1 -> 9.9.  It takes three stages: with the two that eight rows of 4096 channels leave, 32000
// rows gain nothing.  Nine to sixteen rows (a second set of products, fewer stages) from 100 M
// weights on: 151936 x 2560 72 to 74 us against 81 to 83 in the form above, 40000 x 2560 28 both,
// 19456 x 2560 20 against 18.
constexpr int STREAM_ROWS = 16, STREAM_MAX = 8;

inline int w8_stream_stages(int M, int K) {
  const size_t row = K + 64;
  const size_t rows = M * row;
  const size_t fit = rows > GEMV_SMEM_LIMIT ? 0 : (GEMV_SMEM_LIMIT - rows) / (STREAM_ROWS * row);
  return static_cast<int>(fit < STREAM_MAX ? fit : STREAM_MAX);
}

inline bool w8_streams(int M, int N, int K) {
  return w8_stream_stages(M, K) >= 3 &&
         static_cast<long long>(N) * K >= (M > 8 ? 100000000 : 24000000);
}

template <int PLANES>                                      // of eight activation rows
__global__ void __launch_bounds__((1 + STREAM_MAX) * 32) w8_stream_kernel(
    const int8_t* a, const float* a_scale, const int8_t* w, const __half* w_scale,
    void* __restrict__ out, int M, int N, int K, int out_f32, int stages, int* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[STREAM_MAX], empty[STREAM_MAX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int stride = K + 64, tiles = (N + STREAM_ROWS - 1) / STREAM_ROWS;
  unsigned char* act = smem_raw;                           // [M][stride]
  unsigned char* ring = smem_raw + M * stride;             // [stages][16][stride]
  const int count = (tiles - static_cast<int>(blockIdx.x) + gridDim.x - 1) / gridDim.x;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_fence_init();
  }
  grid_wait();
  grid_release();
  for (int c = threadIdx.x; c < M * (K / 16); c += blockDim.x) {
    const int m = c / (K / 16), k = (c - m * (K / 16)) * 16;
    *reinterpret_cast<int4*>(act + m * stride + k) =
        *reinterpret_cast<const int4*>(a + static_cast<size_t>(m) * K + k);
  }
  __syncthreads();
  if (warp == 0) {
    int issued = 0;
    for (int i = 0; i < count; ++i) {
      const int s = i % stages;
      const bool ok = mbar_wait(&empty[s], ((i / stages) & 1) ^ 1, status, STATUS_TMA_WAIT, i);
      if (!__all_sync(0xffffffffu, ok)) break;
      const int n0 = (blockIdx.x + i * gridDim.x) * STREAM_ROWS, rows = min(STREAM_ROWS, N - n0);
      if (lane == 0) mbar_expect_tx(&full[s], rows * K);
      __syncwarp();
      if (lane < rows)
        bulk_load(ring + static_cast<size_t>(s * STREAM_ROWS + lane) * stride,
                  w + static_cast<size_t>(n0 + lane) * K, K, &full[s]);
      issued = i + 1;
    }
    // no copy of ours is in flight when the CTA ends
    for (int i = max(0, issued - stages); i < issued; ++i)
      mbar_wait(&full[i % stages], (i / stages) & 1, status, STATUS_TMA_WAIT, 0x4000);
    return;
  }
  const int s = warp - 1;
  float sa[PLANES][2];
  const unsigned char* brow[PLANES];
  bool live[PLANES];                                       // columns past the last row are zero
#pragma unroll
  for (int p = 0; p < PLANES; ++p) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
      sa[p][e] = 8 * p + 2 * t + e < M ? a_scale[8 * p + 2 * t + e] : 0.f;
    live[p] = 8 * p + g < M;
    brow[p] = act + min(8 * p + g, M - 1) * stride + t * 16;
  }
  const unsigned char* r0 = ring + static_cast<size_t>(s * STREAM_ROWS + g) * stride + t * 16;
  const unsigned char* r1 = r0 + 8 * stride;
  for (int i = s; i < count; i += stages) {
    const int n = (blockIdx.x + i * gridDim.x) * STREAM_ROWS + g;
    const float w0 = n < N ? __half2float(w_scale[n]) : 0.f;
    const float w1 = n + 8 < N ? __half2float(w_scale[n + 8]) : 0.f;
    const bool ok = mbar_wait(&full[s], (i / stages) & 1, status, STATUS_DECODE_WAIT, i);
    if (!__all_sync(0xffffffffu, ok)) break;
    int acc[PLANES][2][4] = {};
#pragma unroll 4
    for (int k = 0; k < K; k += 64) {
      const uint4 x = *reinterpret_cast<const uint4*>(r0 + k);
      const uint4 y = *reinterpret_cast<const uint4*>(r1 + k);
#pragma unroll
      for (int p = 0; p < PLANES; ++p) {
        uint4 b = make_uint4(0, 0, 0, 0);
        if (live[p]) b = *reinterpret_cast<const uint4*>(brow[p] + k);
        mma_i8_16832(acc[p][0], x.x, y.x, x.y, y.y, b.x, b.y);
        mma_i8_16832(acc[p][1], x.z, y.z, x.w, y.w, b.z, b.w);
      }
    }
    // every word of the tile went into one of these two chains of sums
    hand_back(&empty[s], static_cast<uint32_t>(acc[0][0][0] ^ acc[0][1][0]));
#pragma unroll
    for (int p = 0; p < PLANES; ++p)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 8 * p + 2 * t + (e & 1), at = n + (e >> 1) * 8;
        if (m < M && at < N)
          store_row<1>(out, out_f32, m, at, N, acc[p][0][e] + acc[p][1][e], e >> 1 ? w1 : w0,
                       sa[p][e & 1]);
      }
  }
}

// ---------------------------------------------------------------- experts with few rows each
// Grouped form for decode batches: the tile table of the MoE plan lists (expert, first row, rows),
// most experts have one or two rows, and the tensor-core GEMM would spend a 128-row tile on
// each.  Here a warp takes one (tile, 16-row group of its expert's bank) item at a time over the
// whole K, weights as A and up to eight activation rows as B as above; the activations are read
// from global memory with the weights (a tile's rows are shared by the warps of a CTA through
// L1).  Tiles of more rows repeat the decode once per sixteen rows.
constexpr int GROUPED_CTAS = 148;

__device__ __forceinline__ int warp_scan(int v) {              // sums of lanes 0..l
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) >= static_cast<unsigned>(o)) v += up;
  }
  return v;
}

template <int FMT>
struct ExpertUnit {
  GemvUnit<FMT> u;
  uint4 act[2];                                    // this lane's 32 bytes of activation row g
};

// MIXED takes the tiles of at most most_rows rows and leaves the others to another kernel.
template <int FMT, bool MIXED>
__global__ void __launch_bounds__(GEMV_THREADS, 1) qgemv_grouped_kernel(
    const int8_t* a, const float* a_scale, const unsigned char* w, const __half* w_scale,
    __half* __restrict__ out, int N, int K, long long bank_bytes,
    const E8pTables* __restrict__ tables, const int* tiles, const int* meta, int most_rows,
    int listed) {
  using W = GemvUnit<FMT>;
  constexpr int NB = 2;                            // eight-row blocks per pass over the weights
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int WARPS = GEMV_THREADS / 32;
  int(*red)[NB * 5][32] = reinterpret_cast<int(*)[NB * 5][32]>(
      smem_raw + (FMT == 0 ? 0 : sizeof(E8pRows)));    // [WARPS]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t lane4 = lane * 4;
  // MIXED lists its tiles in shared memory before the tables are filled: there may be none.
  E8pFill<GEMV_THREADS> fill;
  if (FMT != 0 && !MIXED) {
    fill.load(tables, tid);
    fill.store(smem_raw, tid);
  }
  grid_wait();
  grid_release();
  int n_tiles = meta[0];
  const int* list = nullptr;
  if (MIXED && most_rows > 0) {
    int* found = reinterpret_cast<int*>(&red[WARPS]);
    __shared__ int hits[WARPS];
    int count = 0;
    for (int base = 0; base < n_tiles; base += GEMV_THREADS) {
      const int at = base + tid;
      const bool hit = at < n_tiles && tiles[at * 4 + 2] <= most_rows;
      const unsigned ballot = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) hits[warp] = __popc(ballot);
      __syncthreads();
      const int inc = warp_scan(hits[lane]);                // of the warps up to this lane's
      const int before = __shfl_sync(0xffffffffu, inc, warp) - hits[warp];
      const int slot = count + before + __popc(ballot & ((1u << lane) - 1u));
      if (hit && slot < listed) found[slot] = at;
      count += __shfl_sync(0xffffffffu, inc, 31);
      __syncthreads();
    }
    if (count == 0) return;
    n_tiles = min(count, listed);
    list = found;
    if (FMT != 0) {
      fill.load(tables, tid);
      fill.store(smem_raw, tid);
    }
  }
  __syncthreads();
  const int groups = N / 16, kbs = K / 128, items = n_tiles * groups;
  // With fewer items than warps (a decode step of one or two rows) KS neighbouring warps share
  // an item's K and the first of them adds the parts: the walk over K is a chain of loads.
  // Two share it where whole items would leave a second round to a third of the warps or fewer.
  int ks = 1;
  while (ks < 8 && kbs >= 4 * ks && items * ks * 2 <= static_cast<int>(gridDim.x) * WARPS) ks *= 2;
  if (MIXED) {
    constexpr int ALL = GROUPED_CTAS * WARPS;
    if (kbs >= 4 && items > ALL && items <= ALL + ALL / 3) ks = 2;
  }
  const int sub = warp % ks, kb_lo = kbs * sub / ks, kb_hi = kbs * (sub + 1) / ks;
  const int stride = gridDim.x * (WARPS / ks);
  constexpr int UNIT = FMT == 0 ? 1 : 2, BIAS = FMT == 0 ? 0 : (FMT == 1 ? 75 : 15);
  // byte offset of this lane's two 16-byte pieces inside a 128-channel block of a row
  const int piece0 = FMT == 0 ? t * 16 : t * 32, piece1 = FMT == 0 ? 64 + t * 16 : t * 32 + 16;

  for (int item = blockIdx.x * (WARPS / ks) + warp / ks; item < items; item += stride) {
    const int at = item / groups, n0 = (item - at * groups) * 16;
    const int tile = MIXED && list != nullptr ? list[at] : at;
    const int expert = tiles[tile * 4], first = tiles[tile * 4 + 1];
    const int rows = tiles[tile * 4 + 2];
    const unsigned char* bank = w + static_cast<size_t>(expert) * bank_bytes;
    for (int r0 = 0; r0 < rows; r0 += 8 * NB) {
      const int nb = min(NB, (rows - r0 + 7) / 8);
      // rows past the tile's last one repeat it; their results are not stored
      const int8_t* arow[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b)
        arow[b] = a + static_cast<size_t>(first + min(r0 + b * 8 + g, rows - 1)) * K;
      auto fetch = [&](ExpertUnit<FMT>& v, int kb) {
        if (kb >= kb_hi) return;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = n0 + g + h * 8;
          if (FMT == 0) {
            const uint4* p = reinterpret_cast<const uint4*>(bank) +
                             static_cast<size_t>(n) * (K / 16) + kb * 8 + t;
            const uint4 x = *p, y = p[4];
            v.u.w[h][0] = x.x; v.u.w[h][1] = x.y; v.u.w[h][2 % W::WORDS] = x.z;
            v.u.w[h][3 % W::WORDS] = x.w; v.u.w[h][4 % W::WORDS] = y.x;
            v.u.w[h][5 % W::WORDS] = y.y; v.u.w[h][6 % W::WORDS] = y.z;
            v.u.w[h][7 % W::WORDS] = y.w;
          } else if (FMT == 1) {
            const uint4 x = reinterpret_cast<const uint4*>(
                bank)[(static_cast<size_t>(kb) * N + n) * 4 + t];
            v.u.w[h][0] = x.x; v.u.w[h][1] = x.y;
            v.u.w[h][2 % W::WORDS] = x.z; v.u.w[h][3 % W::WORDS] = x.w;
          } else {
            const uint2 x = reinterpret_cast<const uint2*>(
                bank)[(static_cast<size_t>(kb) * N + n) * 4 + t];
            v.u.w[h][0] = x.x; v.u.w[h][1] = x.y;
          }
        }
        v.act[0] = *reinterpret_cast<const uint4*>(arow[0] + kb * 128 + piece0);
        v.act[1] = *reinterpret_cast<const uint4*>(arow[0] + kb * 128 + piece1);
      };
      int acc[NB][4], asum[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        asum[b] = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[b][e] = 0;
      }
      constexpr int DEPTH = FMT == 0 ? 1 : 2;
      ExpertUnit<FMT> buf[DEPTH];
#pragma unroll
      for (int i = 0; i < DEPTH; ++i) fetch(buf[i], kb_lo + i);
      for (int base = kb_lo; base < kb_hi; base += DEPTH) {
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) {
          const int kb = base + i;
          if (kb >= kb_hi) break;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t f[4];                         // {row g, row g + 8} x {low, high} words
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (FMT == 0) {
                f[h] = buf[i].u.w[h][(2 * j) % W::WORDS];
                f[2 + h] = buf[i].u.w[h][(2 * j + 1) % W::WORDS];
              } else {
                const uint32_t word = buf[i].u.w[h][(FMT == 1 ? j : j >> 1) % W::WORDS];
                const uint2 v = FMT == 1 ? e8p_bytes_q4(word, smem_raw, lane4)
                                : j & 1  ? e8p_bytes_q2<1>(word, smem_raw, lane4)
                                         : e8p_bytes_q2<0>(word, smem_raw, lane4);
                f[h] = v.x;
                f[2 + h] = v.y;
              }
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              uint32_t x0, x1;
              if (b == 0) {
                const uint4& p = buf[i].act[j >> 1];
                x0 = j & 1 ? p.z : p.x;
                x1 = j & 1 ? p.w : p.y;
              } else {
                if (b >= nb) break;
                const uint2 p = *reinterpret_cast<const uint2*>(
                    arow[b] + kb * 128 + (j >> 1 ? piece1 : piece0) + (j & 1) * 8);
                x0 = p.x;
                x1 = p.y;
              }
              if (FMT != 0)
                asum[b] = __dp4a(static_cast<int>(x1), 0x01010101,
                                 __dp4a(static_cast<int>(x0), 0x01010101, asum[b]));
              mma_i8_16832(acc[b], f[0], f[1], f[2], f[3], x0, x1);
            }
          }
          fetch(buf[i], kb + DEPTH);
        }
      }
      if (ks > 1) {
        // the warps of an item meet at their own named barrier, before and after the exchange
        if (sub != 0) {
#pragma unroll
          for (int b = 0; b < NB; ++b) {
#pragma unroll
            for (int e = 0; e < 4; ++e) red[warp][b * 5 + e][lane] = acc[b][e];
            red[warp][b * 5 + 4][lane] = asum[b];
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(warp / ks), "r"(ks * 32) : "memory");
        if (sub == 0) {
          for (int q = 1; q < ks; ++q) {
#pragma unroll
            for (int b = 0; b < NB; ++b) {
#pragma unroll
              for (int e = 0; e < 4; ++e) acc[b][e] += red[warp + q][b * 5 + e][lane];
              asum[b] += red[warp + q][b * 5 + 4][lane];
            }
          }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(warp / ks), "r"(ks * 32) : "memory");
        if (sub != 0) continue;
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (b >= nb) break;
        asum[b] += __shfl_xor_sync(0xffffffffu, asum[b], 1);
        asum[b] += __shfl_xor_sync(0xffffffffu, asum[b], 2);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int m = r0 + b * 8 + 2 * t + (e & 1), n = n0 + g + (e >> 1) * 8;
          const int sum = __shfl_sync(0xffffffffu, asum[b], (2 * t + (e & 1)) * 4);
          if (m < rows) {
            const int total = UNIT * acc[b][e] - BIAS * sum;
            const float sw = __half2float(w_scale[static_cast<size_t>(expert) * N + n]);
            out[static_cast<size_t>(first + m) * N + n] =
                __float2half_rn((static_cast<float>(total) * sw) * a_scale[first + m]);
          }
        }
      }
    }
  }
}

template <int FMT, bool MIXED>
static int launch_grouped(const int8_t* a, const float* as, const void* w, const __half* ws,
                          void* out, int N, int K, long long bank, const int* tiles,
                          const int* meta, int most_rows, int max_tiles, cudaStream_t stream) {
  const int listed = most_rows > 0 ? max_tiles : 0;
  const size_t smem = (FMT == 0 ? 0 : sizeof(E8pRows)) +
                      (static_cast<size_t>(GEMV_THREADS) * 10 + listed) * sizeof(int);
  if (smem > GEMV_SMEM_LIMIT) return -1;
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, qgemv_grouped_kernel<FMT, MIXED>,
                                       MIXED ? GEMV_SMEM_LIMIT : smem))
    return e;
  launch_early(qgemv_grouped_kernel<FMT, MIXED>, GROUPED_CTAS, GEMV_THREADS, smem, stream, a, as,
               reinterpret_cast<const unsigned char*>(w), ws, reinterpret_cast<__half*>(out), N,
               K, bank, runtime_e8p_tables(), tiles, meta, most_rows, listed);
  return static_cast<int>(cudaGetLastError());
}

int qgemv_grouped_dispatch(int fmt, const int8_t* a, const float* as, const void* w,
                           const __half* ws, void* out, int N, int K, long long bank,
                           const int* tiles, const int* meta, int most_rows, int max_tiles,
                           cudaStream_t stream) {
  // INT8 has the one form for both: its loop comes out better with the list (128 experts of 1536 x
  // 2048, 14 skewed rows: 31 us against 36); the E8P forms pay 0.4 us of 6 for it.
  const bool mixed = most_rows > 0;
  const auto run = fmt == 0   ? launch_grouped<0, true>
                   : fmt == 1 ? (mixed ? launch_grouped<1, true> : launch_grouped<1, false>)
                              : (mixed ? launch_grouped<2, true> : launch_grouped<2, false>);
  return run(a, as, w, ws, out, N, K, bank, tiles, meta, most_rows, max_tiles, stream);
}

// Grid shape: n_parts x k_parts CTAs on the 148 SMs.  E8P projections may split K (2, 4 or 8
// ways, at least 4 k-blocks each) when their rows divide badly over the SMs.  The costs are
// measured: 0.03 us per eight rows x 128 channels on a full SM (Q4; 19456 x 2560: 16.4 x 20 of
// them in 10 us), and about 2.5 us for the round trip through the workspace, which is why
// splitting pays for long K only (2560 x 4096 took 10.3 us in eight parts, 6.7 us for a 2048 x
// 4096 projection unsplit).
struct GemvGrid {
  int n_parts, k_parts, max_groups;
};
static GemvGrid gemv_grid(int fmt, int N, int K) {
  const int oct = N / 8, kb = K / 128;
  GemvGrid best{1, 1, 0};
  if (fmt == 0) {
    best.n_parts = oct < 148 ? oct : 148;
  } else {
    double best_cost = 0.0;
    for (int kp = 1; kp <= 8; kp *= 2) {
      if (kp > 1 && (kb / kp < 4 || N > GEMV_WS_COLS || 148 / kp > GEMV_WS_TICKETS)) break;
      const int np = oct < 148 / kp ? oct : 148 / kp;
      const double cost = ((oct + np - 1) / np) * ((kb + kp - 1) / kp) * (fmt == 1 ? 0.03 : 0.02) +
                          (kp > 1 ? 2.5 : 0.0);
      if (kp == 1 || cost < best_cost) {
        best_cost = cost;
        best = GemvGrid{np, kp, 0};
      }
    }
  }
  best.max_groups = ((oct + best.n_parts - 1) / best.n_parts + 1) / 2;
  return best;
}

// Whether an E8P projection runs on e8p_dp4a_kernel: where it was the quicker of the two, over 250
// to 19456 columns x 1024 to 9728 channels, alone and with each row preparation.
//   alone: Q4 one or two rows always (1 x 19456 x 2560 13.4 us against 14.9); four rows under short
//     or narrow products (2048 x 1024 6.1 against 7.2, 9728 x 2048 10.2 against 10.6, 5120 x 4096
//     11.1 against 10.7), eight under small ones (2048 x 1024 6.9 against 7.7, 2560 x 1024 both
//     7.7).  Q2 one or two rows from 8 M weights on (2048 x 9728 7.3 against 8.0, 2048 x 2048 both
//     6.2), four and eight rows as for Q4 (4 x 2048 x 4096 7.2 against 7.3, 4 x 2560 x 4096 8.1
//     against 7.9; 8 x 2048 x 2048 7.6 against 7.7, 8 x 5120 x 1024 7.8 against 7.3).
//   with the row preparation, which dominates and leaves the MMA form few registers: always (4 x
//     2048 x 1024 13.4 against 17.7), but for five to eight rows under large products of long rows
//     (5 x 19456 x 2560 36.2 against 32.4; 5 x 12288 x 2048 24.8 against 25.9).
inline bool gemv_dp4a(int fmt, int mt, int N, int K, bool fused) {
  const long long cells = static_cast<long long>(N) * K, M = 1024 * 1024;
  if (fused) return mt <= 4 || K <= 2048 || cells < 23 * M;
  if (mt <= 2) return fmt == 1 || cells >= 8 * M;
  if (mt <= 4)
    return (K <= 2048 && cells <= 20 * M) || (fmt == 1 ? N <= 1024 : N <= 2048 && K <= 4096);
  return fmt == 1 ? K <= 1024 && N <= 2048 : K <= 2048 && cells <= 4 * M;
}

// Dynamic shared memory for `mt` staged activation rows.
static size_t gemv_smem(int fmt, int mt, const GemvGrid& g, int K, bool fused) {
  size_t smem = (fmt == 0 ? 0 : sizeof(E8pRows)) + static_cast<size_t>(mt) * K +
                (static_cast<size_t>(g.max_groups) * 16 * (mt + 1) + 2 * mt) * sizeof(int) + 16;
  if (fused) smem += static_cast<size_t>(K) * sizeof(float);
  return smem;
}

template <int FMT, int MT>
static int launch_gemv(const int8_t* a, const float* as, const void* w, const __half* ws, void* out,
                       int M, int N, int K, int out_f32, cudaStream_t stream, const PeerOut& po,
                       const GemvFuse& fz = GemvFuse{}) {
  GemvGrid g = gemv_grid(FMT, N, K);
  size_t smem = gemv_smem(FMT, MT, g, K, fz.pre != 0);
  // very wide INT8 projections under long rows: several waves of CTAs with fewer groups each
  while (FMT == 0 && smem > GEMV_SMEM_LIMIT && g.max_groups > 1) {
    g.n_parts *= 2;
    g.max_groups = ((N / 8 + g.n_parts - 1) / g.n_parts + 1) / 2;
    smem = gemv_smem(FMT, MT, g, K, fz.pre != 0);
  }
  if (smem > GEMV_SMEM_LIMIT) return -1;
  static const int slot[2] = {runtime_new_slot(), runtime_new_slot()};
  auto start = [&](auto kernel, int threads, auto* weights, int sl) -> int {
    if (const int e = runtime_allow_smem(sl, kernel, GEMV_SMEM_LIMIT)) return e;
    const int grid = g.n_parts * g.k_parts;
    // with peers the launch keeps its place behind the kernels before it
    if (po.tp == 0)
      launch_early(kernel, grid, threads, smem, stream, a, as, weights, ws, out, M, N, K, out_f32,
                   runtime_e8p_tables(), po, g.n_parts, g.k_parts, g.max_groups,
                   runtime_gemv_workspace(), fz);
    else
      kernel<<<grid, threads, smem, stream>>>(a, as, weights, ws, out, M, N, K, out_f32,
                                              runtime_e8p_tables(), po, g.n_parts, g.k_parts,
                                              g.max_groups, runtime_gemv_workspace(), fz);
    return static_cast<int>(cudaGetLastError());
  };
  if constexpr (FMT != 0 && MT <= 8)
    if (gemv_dp4a(FMT, MT, N, K, fz.pre != 0))
      return start(e8p_dp4a_kernel<FMT, MT>, Dp4a<FMT, MT>::THREADS, static_cast<const uint4*>(w),
                   slot[0]);
  if constexpr (FMT != 1 || MT > 2) return start(qgemv_kernel<FMT, MT>, GEMV_THREADS, w, slot[1]);
  return -1;
}

template <int MT>
static int launch_w8(const int8_t* a, const float* as, const void* w, const __half* ws, void* out,
                     int M, int N, int K, int out_f32, cudaStream_t stream, const PeerOut& po) {
  const size_t smem = static_cast<size_t>(MT) * K;
  if (smem > 200 * 1024) return -1;
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, w8_gemv_kernel<MT>, 200 * 1024)) return e;
  const int grid = (N + W8_WARPS - 1) / W8_WARPS;
  const int8_t* weights = reinterpret_cast<const int8_t*>(w);
  if (po.tp == 0)
    launch_early(w8_gemv_kernel<MT>, grid, W8_WARPS * 32, smem, stream, a, as, weights, ws, out,
                 M, N, K, out_f32, po);
  else
    w8_gemv_kernel<MT><<<grid, W8_WARPS * 32, smem, stream>>>(a, as, weights, ws, out, M, N, K,
                                                              out_f32, po);
  return static_cast<int>(cudaGetLastError());
}

static int launch_w8_stream(const int8_t* a, const float* as, const void* w, const __half* ws,
                            void* out, int M, int N, int K, int out_f32, cudaStream_t stream) {
  const int stages = w8_stream_stages(M, K);
  const size_t smem = static_cast<size_t>(K + 64) * (M + stages * STREAM_ROWS);
  static const int slot[2] = {runtime_new_slot(), runtime_new_slot()};
  auto kernel = M > 8 ? w8_stream_kernel<2> : w8_stream_kernel<1>;
  if (const int e = runtime_allow_smem(slot[M > 8], kernel, GEMV_SMEM_LIMIT)) return e;
  const int tiles = (N + STREAM_ROWS - 1) / STREAM_ROWS;
  launch_early(kernel, tiles < 148 ? tiles : 148, (1 + stages) * 32, smem, stream, a,
               as, reinterpret_cast<const int8_t*>(w), ws, out, M, N, K, out_f32, stages,
               runtime_status_ptr());
  return static_cast<int>(cudaGetLastError());
}

int qgemv_dispatch(int fmt, const int8_t* a, const float* as, const void* w, const __half* ws,
                   void* out, int M, int N, int K, int out_f32, cudaStream_t stream,
                   const PeerOut* peer) {
  PeerOut po{};
  if (peer != nullptr) po = *peer;
  if (M < 1 || M > 8 || K % 128 || N % 8) return -1;
  if (fmt != 0) {
    // Very long rows (K above about 19 000 at eight rows): the staged activations of all
    // rows do not fit beside the tables, so the rows go in several launches.
    int fit = 8;
    const GemvGrid grid = gemv_grid(fmt, N, K);
    while (fit > 1 && gemv_smem(fmt, fit, grid, K, false) > GEMV_SMEM_LIMIT) fit /= 2;
    if (M > fit) {
      if (peer != nullptr && peer->tp > 0) return -1;      // row indices of the push would shift
      const size_t out_row = static_cast<size_t>(N) * (out_f32 ? 4 : 2);
      for (int m0 = 0; m0 < M; m0 += fit) {
        const int rows = M - m0 < fit ? M - m0 : fit;
        const int r = qgemv_dispatch(fmt, a + static_cast<size_t>(m0) * K, as + m0, w, ws,
                                     static_cast<char*>(out) + m0 * out_row, rows, N, K, out_f32,
                                     stream, peer);
        if (r) return r;
      }
      return 0;
    }
  }
#define BY_M(FN, ...)                                            \
  (M == 1 ? FN<__VA_ARGS__ 1>(a, as, w, ws, out, M, N, K, out_f32, stream, po)  \
   : M == 2 ? FN<__VA_ARGS__ 2>(a, as, w, ws, out, M, N, K, out_f32, stream, po) \
   : M <= 4 ? FN<__VA_ARGS__ 4>(a, as, w, ws, out, M, N, K, out_f32, stream, po) \
            : FN<__VA_ARGS__ 8>(a, as, w, ws, out, M, N, K, out_f32, stream, po))
  if (fmt == 0 && po.tp == 0 && w8_streams(M, N, K))
    return launch_w8_stream(a, as, w, ws, out, M, N, K, out_f32, stream);
  if (fmt == 0 && w8_by_rows(M, N, K)) return BY_M(launch_w8, );
  if (fmt == 0)
    return M <= 4 ? launch_gemv<0, 4>(a, as, w, ws, out, M, N, K, out_f32, stream, po)
                  : launch_gemv<0, 8>(a, as, w, ws, out, M, N, K, out_f32, stream, po);
  if (fmt == 1) return BY_M(launch_gemv, 1, );
  if (fmt == 2) return BY_M(launch_gemv, 2, );
#undef BY_M
  return -1;
}

// Nine to sixteen rows take a second set of products over the same decoded weights: exact sums, so
// the bits of the tensor-core GEMM, which decodes a tile for 128 rows however few there are.  Q4,
// sixteen rows: 19456 x 2560 28.2 -> 18.0 us (eight rows 14.6), 12288 x 2048 22.5 -> 12.9, 6144 x
// 2560 12.4 -> 11.2, 1024 x 2048 11.8 -> 8.0; INT8 19456 x 2560 26.2 -> 17.8, 151936 x 2560 as a
// stream 96 -> 74.  Short rows (4096 x 768 5.6 against 7.1) and long ones, whose activations
// fill the shared memory of the one CTA (2560 x 8192 16.3 against 17.2, 2560 x 9728 16.8 against
// 19.7), stay on the tensor cores, as do launches to peers.
bool qgemv_wide(int fmt, int M, int N, int K) {
  if (M <= 8 || M > 16) return false;
  if (fmt == 0 && w8_streams(M, N, K)) return true;
  if (K < 1024 || K > 6144) return false;
  const GemvGrid g = gemv_grid(fmt, N, K);
  if (g.k_parts > 1 && N > GEMV_WS_COLS / 2) return false;
  return fmt == 0 || gemv_smem(fmt, 16, g, K, false) <= GEMV_SMEM_LIMIT;
}
int qgemv_wide_dispatch(int fmt, const int8_t* a, const float* as, const void* w, const __half* ws,
                        void* out, int M, int N, int K, int out_f32, cudaStream_t stream) {
  const PeerOut po{};
  if (fmt == 0 && w8_streams(M, N, K))
    return launch_w8_stream(a, as, w, ws, out, M, N, K, out_f32, stream);
  if (fmt == 0) return launch_gemv<0, 16>(a, as, w, ws, out, M, N, K, out_f32, stream, po);
  if (fmt == 1) return launch_gemv<1, 16>(a, as, w, ws, out, M, N, K, out_f32, stream, po);
  return launch_gemv<2, 16>(a, as, w, ws, out, M, N, K, out_f32, stream, po);
}

// Projection of at most 8 rows with the row preparation fused in (see GemvFuse); E8P weights.
int qgemv_fused_dispatch(int fmt, const void* w, const __half* ws, void* out, int M, int N, int K,
                         cudaStream_t stream, const GemvFuse& fz) {
  if (M < 1 || M > 8 || K % 128 || N % 8 || fz.pre < 1 || fz.pre > 3) return -1;
  if (fmt != 1 && fmt != 2) return -1;
  if (fz.norm_w != nullptr && K / 128 > 128) return -1;
  const PeerOut po{};
#define BY_M(F)                                                                                   \
  (M == 1 ? launch_gemv<F, 1>(nullptr, nullptr, w, ws, out, M, N, K, 0, stream, po, fz)            \
   : M == 2 ? launch_gemv<F, 2>(nullptr, nullptr, w, ws, out, M, N, K, 0, stream, po, fz)          \
   : M <= 4 ? launch_gemv<F, 4>(nullptr, nullptr, w, ws, out, M, N, K, 0, stream, po, fz)          \
            : launch_gemv<F, 8>(nullptr, nullptr, w, ws, out, M, N, K, 0, stream, po, fz))
  if (fmt == 1) return BY_M(1);
  return BY_M(2);
#undef BY_M
}

}  // namespace orinfer

using namespace orinfer;

// pre: 1 = resid (+ x) -> RMSNorm(norm_w) -> rotate(signs) -> A8; 2 = x -> rotate -> A8;
// 3 = SwiGLU(x [M, 2K]) -> rotate -> A8.  out: FP16 [M, N] or null; resid_accum: FP32 [M, N]
// that receives += the FP16-rounded output, or null.  Returns -1 when the shape does not fit
// the fused kernel (more than 8 rows, W8 weights, too much shared memory): the caller then
// uses the separate kernels.
extern "C" int orinfer_qgemv_fused(int fmt, int pre, const __half* x, const float* resid,
                                   const __half* norm_w, const int8_t* signs, float eps,
                                   int zero_centered, int8_t* q_out, float* scale_out,
                                   __half* y_out, const void* w, const __half* w_scale, void* out,
                                   float* resid_accum, int M, int N, int K, cudaStream_t stream) {
  if (runtime_ensure_init() != cudaSuccess) return -2;
  if (pre == 1 && resid == nullptr && x == nullptr) return -1;
  if ((pre == 2 || pre == 3) && x == nullptr) return -1;
  const GemvFuse fz{pre, x, resid, norm_w, signs, eps, zero_centered, q_out, scale_out, y_out,
                    resid_accum};
  return qgemv_fused_dispatch(fmt, w, w_scale, out, M, N, K, stream, fz);
}
