// Causal GQA attention over the paged INT8 KV cache, row-at-a-time form: every query
// row is an independent problem against keys 0..pos of its request, so one kernel
// serves decode (one row per request), MTP verification (a few rows) and chunked
// prefill rows.  The query heads that share a KV head are processed together so the
// INT8 K/V rows are read once; long contexts are split along the key axis into
// partial (max, sum, out) records that a second kernel merges.  Replaces the decode
// configurations of causal_attention_int8 and merge_attention_int8
// (kernels/cuda/model/attention_rows.py:61-276,280-400).
#include "api.h"
#include "common.cuh"
#include "tma.h"

namespace orinfer {

constexpr int ATTN_WARPS = 4;

// Two bytes of `x` (INT8 values plus 128, picked by `sel` from x and 0x64) -> two FP16 values,
// exactly: 0x64xx is 1024 + xx, and 1152 is subtracted.
__device__ __forceinline__ uint32_t int8x2_half2(uint32_t x, uint32_t sel) {
  const uint32_t raw = __byte_perm(x, 0x64646464u, sel);
  const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&raw),
                            __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ uint32_t pack_half2(__half a, __half b) {
  const __half2 v = __halves2half2(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// The G group scales of one cached row, packed as loaded (G = 1: upper half zero).  WIDE: the
// scale tensor is aligned to a whole row of scales.
template <int G, bool WIDE>
struct RowScales {
  uint32_t w[(G + 1) / 2];
  __device__ __forceinline__ void load(const __half* p) {
    if (G == 1 || !WIDE) {
      const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
      for (int i = 0; i < (G + 1) / 2; ++i)
        w[i] = static_cast<uint32_t>(u[2 * i]) |
               (G == 1 ? 0u : static_cast<uint32_t>(u[2 * i + 1]) << 16);
    } else if (G == 2) {
      w[0] = *reinterpret_cast<const uint32_t*>(p);
    } else {
      const uint2 v = *reinterpret_cast<const uint2*>(p);
      w[0] = v.x;
      w[(G + 1) / 2 - 1] = v.y;
    }
  }
  __device__ __forceinline__ float get(int c) const {
    const __half2 v = *reinterpret_cast<const __half2*>(&w[c / 2]);
    return c & 1 ? __high2float(v) : __low2float(v);
  }
  // the scales that `lane` holds
  __device__ __forceinline__ RowScales from(int lane) const {
    RowScales r;
#pragma unroll
    for (int i = 0; i < (G + 1) / 2; ++i) r.w[i] = __shfl_sync(0xffffffffu, w[i], lane);
    return r;
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < (G + 1) / 2; ++i) w[i] = 0u;
  }
};

// One CTA per (row, KV head, key split); its four warps take blocks of KB keys in turn (a block
// lies inside one page) and carry their own softmax state, merged in shared memory at the end.
//
// Both products run on the tensor cores with the INT8 values as exact FP16 integers.
//   S = Q K^T: rows 0..7 of A are the query heads; lane (g, t) reads 16 bytes of key g, which
//   are its B fragments of four steps (the channel order inside a product does not matter, Q
//   is laid out to match).  Each group of 64 channels is summed by itself and scaled in FP32.
//   O = P V: the FP32 weight x value scale is split into an FP16 head and an FP16 remainder
//   in rows g and g + 8 of the same A tile, so the split costs no instruction and keeps 22
//   bits (error against 64 bits as with FP32 products: 2.07e-4 both, the FP16 result's
//   rounding).  The weights are scaled by a power of two (2^14 over the largest value scale seen,
//   exact) so that the remainder stays above the smallest FP16 step.
//
// The first form converted every byte to FP32 and multiplied it once per query head on the CUDA
// cores, with the weights going through shared memory: it was bound by those instructions.  32
// query / 8 KV heads of 128: 128 rows of 320..640 keys 209 -> 53 us with the products on the
// tensor cores and loads through registers, 41 us with the loads in cp.async rings (132 MB: 3.2
// TB/s); 6 rows of 12000..24000 keys 432 -> 78 -> 62 us (235 MB: 3.8 TB/s).  A block's own work
// bounds it: 57 and 62 % of the issue slots and half of the ALU pipe (copies and their addresses,
// scale shuffles, a permute and a subtraction per pair of INT8 values, the head and remainder, two
// maxima per block) with under three warps per scheduler, which wait for fixed latencies and for
// each other; for loads they wait a third of that (0.3 to 0.6 warps per issue).
template <int D>
struct AttnTile {
  static constexpr int G = D / 64;                 // scale groups per row
  static constexpr int KB = D == 256 ? 16 : 32;    // keys per block
  static constexpr int MIN_CTAS = D == 256 ? 2 : D == 128 ? 3 : 4;   // resident per SM
  static constexpr int CPK = D / 16;               // 16-byte units of a key row
  static constexpr int STAGE = 2 * KB * D;         // K and V rows of one block
  static constexpr int RING = ATTN_WARPS * 2 * STAGE;          // two stages per warp
  static constexpr int SMEM = RING > ATTN_WARPS * 8 * D * 4 ? RING : ATTN_WARPS * 8 * D * 4;
  // where 16-byte unit `u` of row `key` of a block lies: the lanes that read together (8 keys
  // x 4 neighbouring units for K; 4 keys x 32 bytes for V) meet on no bank
  __device__ static int k_unit(int key, int u) {
    return key * CPK + (CPK >= 8 ? u ^ ((key & 1) << 2) : u);
  }
  __device__ static int v_unit(int key, int u) {
    return key * CPK + (u ^ (CPK >= 8 ? ((key >> 1) & 3) << 1 : ((key >> 1) & 1) << 1));
  }
};

__device__ __forceinline__ void attn_store(float v, const __half* gate, __half* out, size_t at) {
  if (gate) v *= __fdiv_rn(1.f, 1.f + expf(-__half2float(gate[at])));
  out[at] = __float2half_rn(v);
}

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}

// The four warps' results (R rows of heads each, and the maxima and sums of their weights) become
// the row's output or, where the keys are split, a record for the merge.
template <int D, int R>
__device__ __forceinline__ void attn_finish(const float (*s_o)[R][D], const float (*s_m)[R],
                                            const float (*s_l)[R], bool apart, bool idle, int rep,
                                            int row, int h, int qh, int split, int splits,
                                            const __half* gate, __half* out, float* scratch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (idle) return;
  for (int r = apart ? 0 : warp; r < rep; r += apart ? 1 : ATTN_WARPS) {   // a head per warp
    const size_t head = static_cast<size_t>(row) * qh + h * rep + r;
    float f[ATTN_WARPS], m = apart ? s_m[warp][r] : s_m[0][r], l = apart ? s_l[warp][r] : 0.f;
    if (!apart) {
#pragma unroll
      for (int w = 1; w < ATTN_WARPS; ++w) m = fmaxf(m, s_m[w][r]);
#pragma unroll
      for (int w = 0; w < ATTN_WARPS; ++w) {
        f[w] = s_m[w][r] == -INFINITY ? 0.f : exp2f(s_m[w][r] - m);
        l = fmaf(s_l[w][r], f[w], l);
      }
    }
    float* rec = scratch + (head * splits + split) * (D + 2);
    if (splits > 1 && lane == 0) {
      rec[0] = m;
      rec[1] = l;
    }
#pragma unroll
    for (int d = lane; d < D; d += 32) {
      float o = apart ? s_o[warp][r][d] : 0.f;
      if (!apart) {
#pragma unroll
        for (int w = 0; w < ATTN_WARPS; ++w) o = fmaf(s_o[w][r][d], f[w], o);
      }
      if (splits == 1)
        attn_store(l > 0.f ? o / l : 0.f, gate, out, head * D + d);
      else
        rec[2 + d] = o;
    }
  }
}

// APART: rows of at most apart_keys keys have only a few blocks, of which a warp of a CTA gets one
// or none, and a large launch of them is bound by its waves of CTAs.  Four KV heads then share the
// CTA of the first of them, a warp each, and the other three CTAs return at once.  Used for up to
// as many blocks (four at most) as the launch has waves: a warp then walks them in less time than
// three waves of CTAs take.  16 query / 16 KV heads of 128, 512 rows: about 30 keys 71 -> 33 us,
// 120 keys 87 -> 62; 32 / 8, 128 rows of 64 keys 13.2 -> 12.3, but 64 rows (no second wave) 9.0 ->
// 9.9; fewer than four KV heads leave warps idle (16 / 2 of 256, 512 rows of 60 keys 28 -> 30).
// Longer rows of such a launch pay up to 3 % for the form (8 / 8 of 64, 128 rows of 640 keys).
template <int D, bool WIDE, bool APART>
__global__ void __launch_bounds__(
    ATTN_WARPS * 32, D == 64 && !APART ? 3 : AttnTile<D>::MIN_CTAS) attn_rows_kernel(
    const __half* q, const __half* gate, const int* row_req, const int* row_pos,
    const int* page_table, int max_pages, const int8_t* kc, const int8_t* vc, const __half* ks,
    const __half* vs, __half* __restrict__ out, int qh, int kvh, int splits,
    float* __restrict__ scratch, int rep, int apart_keys) {
  constexpr int G = AttnTile<D>::G, KB = AttnTile<D>::KB;
  constexpr int NT = KB / 8, UT = KB / 16;         // 8-key score tiles, 16-key value tiles
  grid_wait();
  grid_release();
  const int row = blockIdx.x, split = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int kv_len = row_pos[row] + 1;
  const bool apart = APART && kv_len <= apart_keys;
  if (apart && (blockIdx.y & (ATTN_WARPS - 1)) != 0) return;
  const int h = apart ? min(static_cast<int>(blockIdx.y) + warp, kvh - 1) : blockIdx.y;
  const bool idle = apart && static_cast<int>(blockIdx.y) + warp >= kvh;
  const int per = (kv_len + splits - 1) / splits;
  const int k_lo = split * per, k_hi = min(kv_len, k_lo + per);
  const int* pages = page_table + static_cast<size_t>(row_req[row]) * max_pages;
  const float qscale = rsqrtf(static_cast<float>(D)) * 1.4426950408889634f;

  using T = AttnTile<D>;
  extern __shared__ __align__(16) unsigned char attn_smem[];   // rings, then the warps' results
  float(*s_o)[8][D] = reinterpret_cast<float(*)[8][D]>(attn_smem);
  __shared__ float s_m[ATTN_WARPS][8], s_l[ATTN_WARPS][8];

  // Query fragments in shared memory, one copy for the four warps of a head (16 or 32 registers per
  // lane buy more loads in flight): halves 4s..4s+3 of a lane's 16 are the A registers of step s.
  __shared__ __align__(16) uint4 s_qs[APART ? ATTN_WARPS : 1][G][2][32];
  uint4(*s_q)[2][32] = s_qs[apart ? warp : 0];
  if (warp == 0 || apart) {
#pragma unroll
    for (int c = 0; c < G; ++c) {
      const __half* p = q + (static_cast<size_t>(row) * qh + h * rep + g) * D + c * 64 + t * 16;
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = 0u;
      if (g < rep) {
        if (WIDE) {
          *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(p);
          *reinterpret_cast<uint4*>(w + 4) = reinterpret_cast<const uint4*>(p)[1];
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) w[i] = pack_half2(p[2 * i], p[2 * i + 1]);
        }
      }
      s_q[c][0][lane] = make_uint4(w[0], w[1], w[2], w[3]);
      s_q[c][1][lane] = make_uint4(w[4], w[5], w[6], w[7]);
    }
  }
  __syncthreads();
  const uint32_t q_addr = smem_u32(&s_q[0][0][lane]);
  float acc[G * 8][4];
#pragma unroll
  for (int i = 0; i < G * 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float m_run = -INFINITY, l_run = 0.f;
  int e_run = -100;                                // the value scales seen are below 2^e_run

  const int step = apart ? 1 : ATTN_WARPS;
  const int b_hi = k_hi > k_lo && !idle ? (k_hi + KB - 1) / KB : 0;
  int b = k_hi > k_lo ? k_lo / KB + (apart ? 0 : warp) : 0;
  // This warp's ring: the block being used and the next one, copied in by cp.async (8 KB in
  // flight per warp without a register).  Lane l also holds the scales of key l of both.
  const uint32_t ring = smem_u32(attn_smem) + warp * 2 * T::STAGE;
  auto first_slot = [&](int blk, int page) {
    return static_cast<size_t>(page) * 128 + ((blk * KB) & 127);
  };
  RowScales<G, WIDE> ks_next, vs_next;
  auto issue = [&](int blk, int page, int st) {
    const size_t slot0 = first_slot(blk, page);
    const int8_t* kp = kc + (slot0 * kvh + h) * D;
    const int8_t* vp = vc + (slot0 * kvh + h) * D;
    const uint32_t dst = ring + st * T::STAGE;
#pragma unroll
    for (int it = 0; it < KB * T::CPK / 32; ++it) {
      const int key = (it * 32 + lane) / T::CPK, u = (it * 32 + lane) % T::CPK;
      const size_t off = static_cast<size_t>(key) * kvh * D + u * 16;
      cp_async16(dst + T::k_unit(key, u) * 16, kp + off);
      cp_async16(dst + KB * D + T::v_unit(key, u) * 16, vp + off);
    }
    const size_t cell = ((slot0 + (lane & (KB - 1))) * kvh + h) * G;
    ks_next.load(ks + cell);
    vs_next.load(vs + cell);
  };
  // the page id of a block is fetched two blocks ahead
  int page_next = b + step < b_hi ? pages[((b + step) * KB) >> 7] : 0;
  if (b < b_hi) issue(b, pages[(b * KB) >> 7], 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int st = 0; b < b_hi; b += step, st ^= 1) {
    const int key0 = b * KB;
    RowScales<G, WIDE> ks_cur = ks_next, vs_cur = vs_next;
    if (b + step < b_hi) {
      issue(b + step, page_next, st ^ 1);
      if (b + 2 * step < b_hi) page_next = pages[((b + 2 * step) * KB) >> 7];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const uint32_t k_s = ring + st * T::STAGE, v_s = k_s + KB * D;
    // scales of this lane's keys 8 i + 2 t + e
    RowScales<G, WIDE> vsc[UT][4], ksc[NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        ksc[i][e] = ks_cur.from(8 * i + 2 * t + e);
        vsc[i >> 1][(i & 1) * 2 + e] = vs_cur.from(8 * i + 2 * t + e);
      }
    // ---- scores: lane (g, t) gets head g against keys 8 i + 2 t and 8 i + 2 t + 1
    float s[NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i) s[i][0] = s[i][1] = 0.f;
#pragma unroll
    for (int c = 0; c < G; ++c) {
      uint32_t qf[8];
#pragma unroll
      for (int j = 0; j < 2; ++j)                     // volatile: not hoisted into registers
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(qf[4 * j]), "=r"(qf[4 * j + 1]), "=r"(qf[4 * j + 2]),
                       "=r"(qf[4 * j + 3])
                     : "r"(q_addr + (c * 2 + j) * 512));
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t w[4];
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                     : "r"(k_s + T::k_unit(i * 8 + g, c * 4 + t) * 16));
#pragma unroll
        for (int st = 0; st < 4; ++st) {
          const uint32_t x = w[st] ^ 0x80808080u;
          mma16816(d, qf[2 * st], 0u, qf[2 * st + 1], 0u, int8x2_half2(x, 0x4140),
                   int8x2_half2(x, 0x4342));
        }
        s[i][0] = fmaf(d[0], ksc[i][0].get(c), s[i][0]);
        s[i][1] = fmaf(d[1], ksc[i][1].get(c), s[i][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      s[i][0] *= qscale;
      s[i][1] *= qscale;
    }
    if (key0 < k_lo || key0 + KB > k_hi) {
      // keys outside the split: no weight, and their (possibly never written) scales unused
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = key0 + i * 8 + 2 * t + e;
          if (key < k_lo || key >= k_hi) {
            s[i][e] = -INFINITY;
            vsc[i >> 1][(i & 1) * 2 + e].clear();
          }
        }
    }
    // ---- softmax state
    float mb = s[0][0], vmax = 0.f;
#pragma unroll
    for (int i = 0; i < NT; ++i) mb = fmaxf(mb, fmaxf(s[i][0], s[i][1]));
#pragma unroll
    for (int u = 0; u < UT; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < G; ++c) vmax = fmaxf(vmax, fabsf(vsc[u][e].get(c)));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, 1));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, 2));
    const int e_new = max(e_run, static_cast<int>(__float_as_uint(vmax) >> 23) - 126);
    const float m_new = fmaxf(m_run, mb);
    const float corr = m_run == -INFINITY ? 0.f : exp2f(m_run - m_new);
    const bool same = m_new == m_run && e_new == e_run;
    if (!__all_sync(0xffffffffu, same)) {
      const float f =
          corr * __uint_as_float(static_cast<uint32_t>(127 + max(e_run - e_new, -126)) << 23);
#pragma unroll
      for (int i = 0; i < G * 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] *= f;
    }
    m_run = m_new;
    e_run = e_new;
    const float unit = __uint_as_float(static_cast<uint32_t>(127 + 14 - e_new) << 23);
    float lsum = 0.f;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[i][e] = exp2f(s[i][e] - m_new);
        lsum += s[i][e];
      }
    l_run = fmaf(l_run, corr, lsum);
    // ---- values
#pragma unroll
    for (int u = 0; u < UT; ++u) {
#pragma unroll
      for (int c = 0; c < G; ++c) {
        __half hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float p = s[2 * u + (e >> 1)][e & 1] * (vsc[u][e].get(c) * unit);
          hi[e] = __float2half_rn(p);
          lo[e] = __float2half_rn(p - __half2float(hi[e]));
        }
        const uint32_t a0 = pack_half2(hi[0], hi[1]), a1 = pack_half2(lo[0], lo[1]);
        const uint32_t a2 = pack_half2(hi[2], hi[3]), a3 = pack_half2(lo[2], lo[3]);
        uint2 vraw[4];                             // 8 channels of keys 2 t, 2 t + 1 (+ 8)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
                       : "=r"(vraw[e].x), "=r"(vraw[e].y)
                       : "r"(v_s + T::v_unit(u * 16 + 2 * t + (e & 1) + (e >> 1) * 8,
                                             c * 4 + (g >> 1)) * 16 + (g & 1) * 8));
#pragma unroll
        for (int wd = 0; wd < 2; ++wd) {
          uint32_t x[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] = (wd == 0 ? vraw[e].x : vraw[e].y) ^ 0x80808080u;
          // bytes of two keys interleaved: (k0 b0, k1 b0, k0 b1, k1 b1), then b2 and b3
          const uint32_t p01 = __byte_perm(x[0], x[1], 0x5140);
          const uint32_t p23 = __byte_perm(x[0], x[1], 0x7362);
          const uint32_t r01 = __byte_perm(x[2], x[3], 0x5140);
          const uint32_t r23 = __byte_perm(x[2], x[3], 0x7362);
          float(*o)[4] = &acc[c * 8 + wd * 4];
          mma16816(o[0], a0, a1, a2, a3, int8x2_half2(p01, 0x4140), int8x2_half2(r01, 0x4140));
          mma16816(o[1], a0, a1, a2, a3, int8x2_half2(p01, 0x4342), int8x2_half2(r01, 0x4342));
          mma16816(o[2], a0, a1, a2, a3, int8x2_half2(p23, 0x4140), int8x2_half2(r23, 0x4140));
          mma16816(o[3], a0, a1, a2, a3, int8x2_half2(p23, 0x4342), int8x2_half2(r23, 0x4342));
        }
      }
    }
    __syncwarp();                                // the stage is refilled next
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                               // the rings become the result buffers
  // ---- this warp's result: head + remainder rows, back to the unscaled weights
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  const float back = __uint_as_float(static_cast<uint32_t>(127 + max(e_run - 14, -126)) << 23);
  if (g < rep) {
#pragma unroll
    for (int c = 0; c < G; ++c)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        float* dst = &s_o[warp][g][c * 64 + (2 * t + n) * 8];
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          float4 v;
          v.x = (acc[c * 8 + j][n] + acc[c * 8 + j][n + 2]) * back;
          v.y = (acc[c * 8 + j + 1][n] + acc[c * 8 + j + 1][n + 2]) * back;
          v.z = (acc[c * 8 + j + 2][n] + acc[c * 8 + j + 2][n + 2]) * back;
          v.w = (acc[c * 8 + j + 3][n] + acc[c * 8 + j + 3][n + 2]) * back;
          *reinterpret_cast<float4*>(dst + j) = v;
        }
      }
    if (t == 0) {
      s_m[warp][g] = m_run;
      s_l[warp][g] = l_run;
    }
  }
  attn_finish<D, 8>(s_o, s_m, s_l, apart, idle, rep, row, h, qh, split, splits, gate, out, scratch);
}

// ---------------------------------------------------------------- digit form
// The same attention for at most four query heads per KV head, with both products on the INT8
// tensor cores and no conversion of what the cache holds.
//   S = Q K^T: the query, FP16, becomes a fixed-point number of 31 bits under a power of two per
//   head and group of 64 channels, and that four signed digits to the base 256; rows 4 i + r of A
//   are digit i (the largest first) of head r.  INT32 sums over a group are exact, and the digits'
//   sums meet in FP32.
//   O = P V: the FP32 weight x value scale becomes a fixed-point number of 32 bits, four digits,
//   in the same rows, and the sums stay in INT32 accumulators from block to block.
// The weights are relative to a power of two per head, which follows the row's maximum when that is
// more than 2^DIGIT_LAG above it.  The products with the value scales have a unit per head and
// group of 64 channels, in which the largest of them so far takes 27 to 31 bits: one that has
// outgrown its unit shows in its first digit, and only then is the unit chosen anew, for the
// largest product of the block, and the group's accumulators are rescaled, in place.  (Under one
// unit for all heads, groups and keys, above the largest value scale, a group of scales 2^-k of the
// others lost k bits, and so did all keys beside one with a large scale and no weight.)  A query
// value is exact down to 2^-19 of its group's largest and rounded at 2^-31 of that below it.
// Error against 64 bits ahead of the output's FP16 rounding (2.07e-4): 8 rows of 900 keys 1.7e-7
// (the form above 1.8e-7), 3 rows of 20000 2.1e-7 (2.6e-6), with six times the scores 3.5e-7
// (3.6e-7) and 5.2e-7 (1.2e-6); 4 rows of 900 with one group's value scales 2^-10 of the other's
// 1.7e-7 in that group (1.8e-7, under one unit 2.4e-5), 2^-14 1.7e-7 (2.6e-7, 3.9e-4), with one key
// of 2^10 times the scale and no weight 1.5e-7 (1.7e-7, 6.3e-6).
//
// K and V come by TMA as they lie in the cache, a box of 32 keys each, swizzled for ldmatrix; V's
// fragments are transposed by the load (m16n16 b8).  A lane owns eight keys of a block in both
// products; which ones is chosen so that neither side's loads meet on a bank.
//
// A block of 32 keys is 520 instructions of a warp where the form above takes 1060 (counted between
// 4096 and 8192 keys), and a warp of a CTA has 930 besides.  32 / 8 heads of 128: 6 rows of
// 12000..24000 keys 62.7 -> 49.8 us (235 MB; the blocks alone run at the memory's rate), 38 rows of
// 1500..3000 57.5 -> 39.4, 128 rows of 320..640 38.7 -> 33.9.  (A unit that gives the largest
// product one bit more is outgrown so often that the last takes 34.4.)  It is 2.3 waves of CTAs,
// each of which waits 4000 cycles for its row, pages and first block and takes 3000 to finish
// besides the 12000 of its blocks: 39 % of the issue slots, a warp waits 1.7 cycles an instruction
// for the one before it, 1.4 for shared memory, exchanges and conversions, 1.1 for loads.  Tried:
// blocks of 64 keys with one buffer (the same), the heads of a row side by side in the grid (the
// same, long rows 4 % slower), a warp per row of up to 512 keys (the same with 128 rows, 64 rows
// 28.4 against 21.8), scales by loads into registers (the loop's move waits for them: the same,
// long rows 2 % quicker), two products to an instruction (128 rows 5 % slower).
template <int D>
struct DigitTile {
  static constexpr int G = D / 64, KB = 32, KSTEPS = D / 32;
  static constexpr int ROWS = KB * D;                    // K or V of one block
  static constexpr int STAGES = 2;
  static constexpr int RING = ATTN_WARPS * STAGES * 2 * ROWS;
  static constexpr int SMEM = RING + 1024;
  static constexpr int MIN_CTAS = D == 128 ? 3 : 4;
  // 16-byte unit `u` of row `key`: the hardware's 128- or 64-byte swizzle
  __device__ static uint32_t unit(int key, int u) {
    return key * D + ((D == 128 ? u ^ (key & 7) : u ^ ((key >> 1) & 3)) << 4);
  }
  // The key of a 16-key half block that lane t of a quad owns as its number x (0..3): 2t, 2t + 1
  // and two of the upper eight, rotated so that the eight rows that a load reads together (all t
  // with one x pair for K, two t with all x for V) differ modulo 8.
  __device__ static int key_of(int t, int x) {
    return x < 2 ? 2 * t + x : 8 + ((2 * t + 4 + (x & 1)) & 7);
  }
};
constexpr float DIGIT_LAG = 8.f;                         // of the weights' reference, binades
constexpr int DIGIT_BITS = 27;                           // of the product that a unit is chosen for
constexpr int DIGIT_UNIT_MAX = 100;                      // units are at most 2^this and begin so
// Keys of a warp after which the accumulators are scaled down: a digit's sum grows by at most
// 128 x 127 a key.
constexpr int DIGIT_BLOCKS = (1 << 16) / 32;

__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float two_to(int e) {         // e in -126..127
  return __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
}

// the scales of two neighbouring keys
template <int G>
__device__ __forceinline__ void load_pair(float (&v)[2 * G], const float* p) {
  if (G == 2) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2 * G - 2] = x.z; v[2 * G - 1] = x.w;
  } else {
    const float2 x = *reinterpret_cast<const float2*>(p);
    v[0] = x.x; v[1] = x.y;
  }
}

template <int D, bool APART>
__global__ void __launch_bounds__(ATTN_WARPS * 32, DigitTile<D>::MIN_CTAS) attn_digits_kernel(
    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
    const __half* q, const __half* gate, const int* row_req, const int* row_pos,
    const int* page_table, int max_pages, const __half* ks, const __half* vs,
    __half* __restrict__ out, int qh, int kvh, int splits, float* __restrict__ scratch, int rep,
    int apart_keys, int* status) {
  using T = DigitTile<D>;
  constexpr int G = T::G, KB = T::KB, KSTEPS = T::KSTEPS;
  grid_wait();
  grid_release();
  const int row = blockIdx.x, split = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, upper = lane >> 4, head = g & 3;
  const int kv_len = row_pos[row] + 1;
  const bool apart = APART && kv_len <= apart_keys;
  if (apart && (blockIdx.y & (ATTN_WARPS - 1)) != 0) return;
  const int h = apart ? min(static_cast<int>(blockIdx.y) + warp, kvh - 1) : blockIdx.y;
  const bool idle = apart && static_cast<int>(blockIdx.y) + warp >= kvh;
  const int per = (kv_len + splits - 1) / splits;
  const int k_lo = split * per, k_hi = min(kv_len, k_lo + per);
  const int* pages = page_table + static_cast<size_t>(row_req[row]) * max_pages;

  extern __shared__ unsigned char digits_smem[];
  unsigned char* smem = digits_smem + ((1024u - (smem_u32(digits_smem) & 1023u)) & 1023u);
  float(*s_o)[4][D] = reinterpret_cast<float(*)[4][D]>(smem);   // the warps' results, at the end
  __shared__ float s_m[ATTN_WARPS][4], s_l[ATTN_WARPS][4];
  __shared__ __align__(16) uint4 s_q[KSTEPS][32];
  // scales of two blocks, K's and V's: [pair of keys][group][key of the pair]
  __shared__ __align__(16) float s_scale[ATTN_WARPS][2][2][KB / 2][G][2];
  __shared__ uint32_t s_raw[ATTN_WARPS][2][2][32];
  __shared__ uint64_t bars[ATTN_WARPS][T::STAGES];
  uint64_t* full = bars[warp];                     // K and V of a stage have landed

  // the query: lane (g, t) holds channels 32 s + 4 t .. and 32 s + 16 + 4 t .. of its head
  const __half* q_at = q + (static_cast<size_t>(row) * qh + h * rep + head) * D + 4 * t;
  uint2 raw[KSTEPS][2];
#pragma unroll
  for (int s = 0; s < KSTEPS; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      raw[s][i] = head < rep ? *reinterpret_cast<const uint2*>(q_at + 32 * s + 16 * i)
                             : make_uint2(0u, 0u);

  // ---- this warp's ring; the first blocks are on their way before the query is looked at
  const int step = apart ? 1 : ATTN_WARPS;
  const int b_hi = k_hi > k_lo && !idle ? (k_hi + KB - 1) / KB : 0;
  const int b0 = k_hi > k_lo ? k_lo / KB + (apart ? 0 : warp) : 0;
  const int mine = b0 < b_hi ? (b_hi - b0 + step - 1) / step : 0;
  // Page ids of this warp's blocks, a lane each, 32 blocks at a time and as many ahead: one that is
  // fetched when it is needed holds up the copies and the scales behind it.
  auto pages_from = [&](int n) {
    return n + lane < mine ? pages[((b0 + (n + lane) * step) * KB) >> 7] : 0;
  };
  int page_ids = pages_from(0), page_ids_next = pages_from(32);
  unsigned char* ring = smem + warp * T::STAGES * 2 * T::ROWS;
  auto issue = [&](int n, int page) {              // one lane
    unsigned char* to = ring + (n & 1) * 2 * T::ROWS;
    const int slot = page * 128 + (((b0 + n * step) * KB) & 127);
    mbar_expect_tx(&full[n & 1], 2 * T::ROWS);
    tma_load_3d(to, &tmap_k, &full[n & 1], 0, h, slot);
    tma_load_3d(to + T::ROWS, &tmap_v, &full[n & 1], 0, h, slot);
  };
  // The scales of key `lane` of a block as they lie in the cache, two blocks ahead of their use: by
  // cp.async, since a load into a register that the loop moves on is waited for there.  One group's
  // two bytes come with a neighbour's (the slots are an even number).
  const uint32_t raw_u = smem_u32(&s_raw[warp][0][0][lane]);
  auto fetch_scales = [&](int n, int page) {
    const size_t slot =
        static_cast<size_t>(page) * 128 + (((b0 + n * step) * KB) & 127) + lane;
    const size_t at = (slot * kvh + h) * G & ~static_cast<size_t>(1);
    const uint32_t to = raw_u + (n & 1) * 256;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(ks + at) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + 128), "l"(vs + at)
                 : "memory");
  };
  {
    const int page0 = __shfl_sync(0xffffffffu, page_ids, 0);
    const int page1 = __shfl_sync(0xffffffffu, page_ids, 1);
    if (lane == 0) {
      for (int i = 0; i < T::STAGES; ++i) mbar_init(&full[i], 1);
      mbar_fence_init();
      if (mine > 0) issue(0, page0);
      if (mine > 1) issue(1, page1);
    }
    if (mine > 0) fetch_scales(0, page0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (mine > 1) fetch_scales(1, page1);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // ---- its digits: rows g and g + 8 of A are digits `upper` and 2 + `upper`
  const uint32_t sel = upper ? 0x4062u : 0x5173u;  // their bytes in two numbers
  float f_head[G];                                 // the unit of the second one's sums
  uint32_t qa[KSTEPS][4];
#pragma unroll
  for (int c = 0; c < G; ++c) {
    __half2 big2 = __half2half2(__ushort_as_half(0));
#pragma unroll
    for (int s = 2 * c; s < 2 * c + 2; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        big2 = __hmax2_nan(big2, __habs2(reinterpret_cast<const __half2*>(raw[s])[i]));
    __half big_h = __hmax_nan(__low2half(big2), __high2half(big2));
#pragma unroll
    for (int o = 1; o < 4; o <<= 1)
      big_h = __hmax_nan(big_h, __shfl_xor_sync(0xffffffffu, big_h, o));
    const float big = __half2float(big_h);
    const bool finite = big < INFINITY;
    // |q| < 2^e and the fixed-point values below 2^30
    const int e = max(-30, min(16, static_cast<int>(__float_as_uint(big) >> 23) - 126));
    f_head[c] = finite ? two_to(e - 30) * (upper ? 1.f : 256.f) : __int_as_float(0x7fc00000);
    const float up = two_to(30 - e);
#pragma unroll
    for (int s = 2 * c; s < 2 * c + 2; ++s) {
      if (!apart && (s & (ATTN_WARPS - 1)) != warp) continue;
      uint32_t(&a)[4] = qa[s];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t u[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          u[j] = static_cast<uint32_t>(__float2int_rn(
                     __half2float(reinterpret_cast<const __half*>(&raw[s][i])[j]) * up)) +
                 0x80808080u;
        const uint32_t p01 = __byte_perm(u[0], u[1], sel), p23 = __byte_perm(u[2], u[3], sel);
        a[2 * i] = __byte_perm(p01, p23, 0x5410) ^ 0x80808080u;
        a[2 * i + 1] = __byte_perm(p01, p23, 0x7632) ^ 0x80808080u;
      }
      if (!apart) s_q[s][lane] = make_uint4(a[0], a[1], a[2], a[3]);
    }
  }
  __syncthreads();
  if (!apart) {
#pragma unroll
    for (int s = 0; s < KSTEPS; ++s) {
      const uint4 v = s_q[s][lane];
      qa[s][0] = v.x; qa[s][1] = v.y; qa[s][2] = v.z; qa[s][3] = v.w;
    }
  }
  // A sum starts at 1.5 x 2^23, so that its bits are those of the float that much larger, and the
  // bias leaves with the factors: (c + bias) w - bias (w + f) + (d + bias) f, exact up to the
  // rounding of a float.
  constexpr int BIAS = 0x4b400000;
  float w_top[G], w_bias[G];
#pragma unroll
  for (int c = 0; c < G; ++c) {
    w_top[c] = f_head[c] * 65536.f;
    w_bias[c] = -12582912.f * (w_top[c] + f_head[c]);
  }

  int acc[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  // per head: the weights are relative to 2^m_ref, a whole power, and the products with the scales
  // of a group to its unit
  float m_ref = -INFINITY, l_run = 0.f;
  float unit[G];
#pragma unroll
  for (int c = 0; c < G; ++c) unit[c] = two_to(DIGIT_UNIT_MAX);
  uint32_t poison = 0u;                            // groups with a value scale that is no number
  bool ok = true;

  // row addresses of this lane: K's rows of tile i are keys 16 (i / 2) + key_of(row / 2, 2 (i % 2)
  // + row % 2), four matrices of 16 bytes; V's are the keys of lane 16 m + 4 t + x
  const uint32_t ring_u = smem_u32(ring);
  const int kn = lane & 7, kt = (lane & 15) >> 2;
  const int k_row[2] = {kn, 8 + ((kn + 4) & 7)};
  const int v_row = 16 * (lane >> 4) + T::key_of(kt, lane & 3);
  const float qscale = rsqrtf(static_cast<float>(D)) * 1.4426950408889634f;

  // The scales of block n, by the lanes that fetched them, a block ahead of their use.
  auto place_scales = [&](int n) {
    const int key = (b0 + n * step) * KB + lane;
    const bool live = key >= k_lo && key < k_hi;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    uint32_t raw[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      raw[w] = *reinterpret_cast<const volatile uint32_t*>(&s_raw[warp][n & 1][w][lane]);
      if (G == 1 && ((lane & kvh) ^ h) & 1) raw[w] >>= 16;        // (a block's first slot is even)
    }
    const __half2 k2 = *reinterpret_cast<const __half2*>(&raw[0]);
    const __half2 v2 = *reinterpret_cast<const __half2*>(&raw[1]);
#pragma unroll
    for (int c = 0; c < G; ++c) {
      // keys outside the split: their (possibly never written) scales unused
      const float kf = live ? (c == 0 ? __low2float(k2) : __high2float(k2)) * qscale : 0.f;
      float vf = live ? (c == 0 ? __low2float(v2) : __high2float(v2)) : 0.f;
      if (!(fabsf(vf) < INFINITY)) {
        poison |= 1u << c;
        vf = 0.f;
      }
      s_scale[warp][n & 1][0][lane >> 1][c][lane & 1] = kf;
      s_scale[warp][n & 1][1][lane >> 1][c][lane & 1] = vf;
    }
  };
  if (mine > 0) place_scales(0);
  int page2 = __shfl_sync(0xffffffffu, page_ids, 2);
  if (mine > 2) fetch_scales(2, page2);
  asm volatile("cp.async.commit_group;" ::: "memory");

  int n = 0;
  for (; n < mine; ++n) {
    const int key0 = (b0 + n * step) * KB, st = n & 1;
    const bool edge = key0 < k_lo || key0 + KB > k_hi;
    ok = warp_all(mbar_wait(&full[st], (n >> 1) & 1, status, STATUS_TMA_WAIT, 0x20));
    if (!ok) break;
    __syncwarp();
    // ---- scores: half m, this lane's key x of it
    const uint32_t k_s = ring_u + st * 2 * T::ROWS, v_s = k_s + T::ROWS;
    float s[2][4];
    uint32_t kb[2][G][4];
    auto load_k = [&](int i) {
#pragma unroll
      for (int c = 0; c < G; ++c)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(kb[i & 1][c][0]), "=r"(kb[i & 1][c][1]), "=r"(kb[i & 1][c][2]),
                       "=r"(kb[i & 1][c][3])
                     : "r"(k_s + T::unit(16 * (i >> 1) + k_row[i & 1], 4 * c + (lane >> 3)))
                     : "memory");
    };
    load_k(0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int d[G][4];
      if (i < 3) load_k(i + 1);
#pragma unroll
      for (int c = 0; c < G; ++c) {
#pragma unroll
        for (int e = 0; e < 4; ++e) d[c][e] = BIAS;
        mma_s8(d[c], qa[2 * c], kb[i & 1][c][0], kb[i & 1][c][1]);
      }
#pragma unroll
      for (int c = 0; c < G; ++c) mma_s8(d[c], qa[2 * c + 1], kb[i & 1][c][2], kb[i & 1][c][3]);
      float kv[2 * G];
      load_pair<G>(kv, s_scale[warp][st][0][8 * (i >> 1) + T::key_of(t, 2 * (i & 1)) / 2][0]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float sum = 0.f;
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const float part = fmaf(__int_as_float(d[c][2 + e]), f_head[c],
                                  fmaf(__int_as_float(d[c][e]), w_top[c], w_bias[c]));
          sum = c == 0 ? part * kv[e] : fmaf(part, kv[2 * c + e], sum);
        }
        s[i >> 1][2 * (i & 1) + e] = sum;
      }
    }
    if (n + 1 < mine) place_scales(n + 1);
    if ((n & 31) == 29) {                          // block n + 3 is the first of the next batch
      page_ids = page_ids_next;
      page_ids_next = pages_from((n | 31) + 33);
    }
    const int page3 = __shfl_sync(0xffffffffu, page_ids, (n + 3) & 31);
    if (n + 3 < mine) fetch_scales(n + 3, page3);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int x = 0; x < 4; ++x) s[m][x] += __shfl_xor_sync(0xffffffffu, s[m][x], 16);
    if (edge) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int key = key0 + 16 * m + T::key_of(t, x);
          if (key < k_lo || key >= k_hi) s[m][x] = -INFINITY;
        }
    }
    // ---- softmax state
    float mb = s[0][0];
#pragma unroll
    for (int i = 1; i < 8; ++i) mb = fmaxf(mb, s[i >> 2][i & 3]);
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
    // `f`: factors of the sums so far.  A reference that moves by whole powers leaves them alone,
    // since the units make up for it.
    float f[G];
#pragma unroll
    for (int c = 0; c < G; ++c) f[c] = 1.f;
    bool rescale = false;
    if (__any_sync(0xffffffffu, mb > m_ref + DIGIT_LAG)) {
      if (mb > m_ref + DIGIT_LAG) {
        const float m_new = ceilf(mb);
        const bool first = m_ref == -INFINITY;
        const int up = static_cast<int>(fminf(m_new - m_ref, 250.f));
        l_run *= ex2_ftz(m_ref - m_new);
#pragma unroll
        for (int c = 0; c < G; ++c) {
          const int was = __float_as_int(unit[c]) >> 23;
          const int now = first ? was : min(was + up, 127 + DIGIT_UNIT_MAX);
          // (where the unit cannot follow as far)
          if (!first && now < was + up) f[c] = __int_as_float(max(127 + now - was - up, 0) << 23);
          rescale = rescale || f[c] != 1.f;
          unit[c] = __int_as_float(now << 23);
        }
        m_ref = m_new;
      }
    }
    if (n > 0 && n % DIGIT_BLOCKS == 0) {
      rescale = true;
#pragma unroll
      for (int c = 0; c < G; ++c) {
        f[c] *= 0.25f;
        unit[c] *= 0.25f;
      }
    }
    float sums[2];                                 // a block's weights first: short chains of sums
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int x = 0; x < 4; ++x) s[m][x] = ex2_ftz(s[m][x] - m_ref);
      sums[m] = (s[m][0] + s[m][1]) + (s[m][2] + s[m][3]);
    }
    l_run += sums[0] + sums[1];
    // The largest product of the block gets DIGIT_BITS bits where it has outgrown its unit.
    auto fit = [&] {
#pragma unroll
      for (int c = 0; c < G; ++c) {
        float big = 0.f;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float w[2 * G];
            load_pair<G>(w, s_scale[warp][st][1][8 * m + T::key_of(t, 2 * i) / 2][0]);
            big = fmaxf(big, fmaxf(fabsf(s[m][2 * i] * w[2 * c]),
                                   fabsf(s[m][2 * i + 1] * w[2 * c + 1])));
          }
        big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
        big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
        if (big * unit[c] >= 1073741824.f) {       // 2^30
          const float now = two_to(DIGIT_BITS + 126 - (__float_as_int(big) >> 23));
          f[c] *= __int_as_float(__float_as_int(now) - __float_as_int(unit[c]) + (127 << 23));
          unit[c] = now;
        }
      }
    };
    uint32_t a[G][4];
    auto digits = [&] {                            // true: a product has outgrown its unit
      uint32_t over = 0u;                          // a top digit of -128: 2^31 or close to it
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        float w[2][2 * G];                         // two pairs of keys
#pragma unroll
        for (int i = 0; i < 2; ++i)
          load_pair<G>(w[i], s_scale[warp][st][1][8 * m + T::key_of(t, 2 * i) / 2][0]);
#pragma unroll
        for (int c = 0; c < G; ++c) {
          uint32_t u[4];
#pragma unroll
          for (int x = 0; x < 4; ++x)
            u[x] = static_cast<uint32_t>(
                       __float2int_rn(s[m][x] * w[x >> 1][2 * c + (x & 1)] * unit[c])) +
                   0x80808080u;
          const uint32_t p01 = __byte_perm(u[0], u[1], sel), p23 = __byte_perm(u[2], u[3], sel);
          const uint32_t top = __byte_perm(p01, p23, 0x5410);
          a[c][2 * m] = top ^ 0x80808080u;
          a[c][2 * m + 1] = __byte_perm(p01, p23, 0x7632) ^ 0x80808080u;
          over |= (top - 0x01010101u) & ~top;
        }
      }
      return !upper && (over & 0x80808080u) != 0u; // (the lower lanes hold the top digits)
    };
    if (n == 0) fit();
    if (__any_sync(0xffffffffu, digits() || rescale) && n > 0) {
      fit();
      // two digits of a sum, 2^16 apart, as one number and back
#pragma unroll
      for (int c = 0; c < G; ++c) {
        if (f[c] == 1.f) continue;
#pragma unroll
        for (int i = 8 * c; i < 8 * c + 8; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float v = fmaf(static_cast<float>(acc[i][e]), 65536.f,
                                 static_cast<float>(acc[i][2 + e])) * f[c];
            const float top = rintf(v * (1.f / 65536.f));
            acc[i][e] = __float2int_rn(top);
            acc[i][2 + e] = __float2int_rn(fmaf(top, -65536.f, v));
          }
      }
      digits();
    }
    // ---- values
    uint32_t vb[2][4];
    auto load_v = [&](int j) {
      asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];"
                   : "=r"(vb[j & 1][0]), "=r"(vb[j & 1][1]), "=r"(vb[j & 1][2]), "=r"(vb[j & 1][3])
                   : "r"(v_s + T::unit(v_row, j))
                   : "memory");
    };
    load_v(0);
#pragma unroll
    for (int j = 0; j < D / 16; ++j) {
      if (j + 1 < D / 16) load_v(j + 1);
      mma_s8(acc[2 * j], a[j / 4], vb[j & 1][0], vb[j & 1][2]);
      mma_s8(acc[2 * j + 1], a[j / 4], vb[j & 1][1], vb[j & 1][3]);
    }
    __syncwarp();
    if (lane == 0 && n + T::STAGES < mine) issue(n + T::STAGES, page2);
    page2 = page3;
  }
  // a warp that gave up waits for what it has in flight
  if (!ok)
    for (int i = n; i < mine && i < n + T::STAGES; ++i)
      mbar_wait(&full[i & 1], (i >> 1) & 1, status, STATUS_TMA_WAIT, 0x22);
  __syncthreads();                               // the rings become the result buffers
  // ---- this warp's result, back to the unscaled weights
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  poison = __reduce_or_sync(0xffffffffu, poison);
  float back[G];
#pragma unroll
  for (int c = 0; c < G; ++c)
    back[c] = poison >> c & 1 ? __int_as_float(0x7fc00000)
                              : __int_as_float((254 << 23) - __float_as_int(unit[c])) *
                                    (upper ? 1.f : 256.f);
#pragma unroll
  for (int j = 0; j < D / 8; ++j) {
    float v[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      v[e] = fmaf(static_cast<float>(acc[j][e]), 65536.f, static_cast<float>(acc[j][2 + e])) *
             back[j / 8];
      v[e] += __shfl_xor_sync(0xffffffffu, v[e], 16);
    }
    if (upper == (j & 1))
      *reinterpret_cast<float2*>(&s_o[warp][head][8 * j + 2 * t]) = make_float2(v[0], v[1]);
  }
  if (lane < 16 && t == 0) {
    s_m[warp][head] = m_ref;
    s_l[warp][head] = l_run;
  }
  attn_finish<D, 4>(s_o, s_m, s_l, apart, idle, rep, row, h, qh, split, splits, gate, out, scratch);
}

// One CTA per row and head.  The records' maxima and sums are read by a lane each and handed round,
// the outputs eight records at a time, since a call of few rows waits for each load in turn: with
// a record per step of the loop, and attn_finish computing every factor anew for each channel, one
// row of 2000 keys and 32 / 8 heads of 128 took 10.7 us (now 8.3), 16 / 2 heads of 256 (32 records)
// 15.1 (10.0), 64 rows of 640 keys unsplit 26.8 (22.9).
template <int D>
__global__ void attn_merge_kernel(
    const float* scratch, const __half* gate, __half* __restrict__ out, int qh, int splits) {
  grid_wait();
  grid_release();
  const int row = blockIdx.x, head = blockIdx.y, lane = threadIdx.x & 31;
  const float* rec = scratch + (static_cast<size_t>(row) * qh + head) * splits * (D + 2);
  float m = -INFINITY;
  for (int s = lane; s < splits; s += 32) m = fmaxf(m, rec[s * (D + 2)]);
  m = warp_max(m);
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float l = 0.f, o = 0.f;
    for (int s0 = 0; s0 < splits; s0 += 32) {
      const int n = min(32, splits - s0);
      const float* own = rec + (s0 + min(lane, n - 1)) * (D + 2);
      const float ms = own[0], ls = own[1];
      const float f = ms == -INFINITY ? 0.f : exp2f(ms - m);
      for (int b = 0; b < n; b += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          v[i] = b + i < n ? rec[(s0 + b + i) * (D + 2) + 2 + d] : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float fs = __shfl_sync(0xffffffffu, f, b + i);
          const float l_s = __shfl_sync(0xffffffffu, ls, b + i);
          if (b + i < n) {
            l = fmaf(l_s, fs, l);
            o = fmaf(v[i], fs, o);
          }
        }
      }
    }
    attn_store(l > 0.f ? o / l : 0.f, gate, out, (static_cast<size_t>(row) * qh + head) * D + d);
  }
}

// Whether a launch of the row kernel may start early.  Of 64 and 128 channels three and more CTAs
// fit an SM, and a grid of more than one and little more than two per SM then gathers where the
// kernel in front ends first, while other SMs get one CTA or none: 32 / 8 heads of 128, contexts of
// 1500 to 3000, 32 rows (256 CTAs) 62 us early and 48 plainly (a decode step of two layers 413 and
// 385), 28 and 37 rows (224, 296) 61 and 62 against 50, 38 rows (304) 63 against 60, 40 rows (320)
// 63 against 64, 17 rows of 3 splits (408) 29 against 32; 128 rows of two KV heads of 256 (256)
// 38.5 against 39.5.
inline bool attn_starts_early(int head_dim, long long ctas) {
  return head_dim > 128 || ctas <= 148 || ctas >= 312;
}

// Up to four query heads per KV head fill the sixteen rows of digits; five and more would take a
// second tile and twice the accumulators, and channels above 128 have no room for theirs.  A CTA
// should have ten blocks or more, counted from the pages of the longest context and one more for
// the keys to come, or where the caller does not know it from the page table's width (a serving
// engine's tables have the width of the longest context there may be): the digits of a query, the
// units of a first block and the sums' way back cost what a few blocks save.  The form above and
// this one, 32 / 8 heads of 128: 1 row of 60 keys 3.5 and 3.7 us, of 900 (68 a CTA) 5.9 and 6.3, 8
// rows of 300 (76) 6.8 and 7.0, of 900 (170) 12.0 and 11.2, of 3000 (512) 19.5 and 17.5, 32 rows of
// 300 10.9 and 10.0, of 3000 48.7 and 37.1.  16 / 8 heads of 64: 16 rows of 60 2.9 and 3.2, of 900
// (341) 10.0 and 10.2, of 3000 (1024) 17.5 and 15.4, 128 rows of 450 21.5 and 19.1.  So the line is
// a compromise: from 150 to 320 keys this form saves 5 % at 128 channels and costs 2 at 64.  Above
// it one kind of call is slower, a little more than a wave of CTAs with contexts of one length: 32
// rows of 900, 32 / 16 heads of 128, 33.5 and 36.2 (ragged ones 30.5 and 27.0).
constexpr int DIGIT_MIN_KEYS = 320;
inline bool attn_digits(int head_dim, int rep, int pages, int splits, bool wide, const void* kc,
                        const void* vc) {
  const long long keys = static_cast<long long>(pages) * 128 / splits;
  return head_dim <= 128 && rep <= 4 && wide && keys >= DIGIT_MIN_KEYS &&
         ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;
}

// The cache as [slots][heads][D] bytes, in boxes of 32 keys of a head.  Which pages are there only
// the page table knows, so the number of slots is left open.
template <int D>
static bool kv_map(CUtensorMap* map, const int8_t* cache, int kvh) {
  PFN_encodeTiled enc = runtime_tma_encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(kvh), 1ull << 31};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(kvh) * D};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(D), 1, 32};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(cache), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             D == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

template <int D>
static int launch_attn(const __half* q, const __half* gate, const int* row_req, const int* row_pos,
                       const int* page_table, int max_pages, const int8_t* kc, const int8_t* vc,
                       const __half* ks, const __half* vs, __half* out, int rows, int qh, int kvh,
                       int rep, int splits, float* scratch, int context, cudaStream_t stream) {
  dim3 grid(rows, kvh, splits);
  const bool wide = ((reinterpret_cast<uintptr_t>(q) & 15) | (reinterpret_cast<uintptr_t>(ks) & 7) |
                     (reinterpret_cast<uintptr_t>(vs) & 7)) == 0;
  const long long ctas = splits > 1 || kvh < ATTN_WARPS ? 0 : static_cast<long long>(rows) * kvh;
  const long long waves = ctas / (148 * AttnTile<D>::MIN_CTAS);
  const int apart_keys = AttnTile<D>::KB * static_cast<int>(waves < 4 ? waves : 4);
  const bool apart = apart_keys > 0;
  if (runtime_ensure_init() != cudaSuccess) return -2;
  const bool early = attn_starts_early(D, static_cast<long long>(rows) * kvh * splits);
  auto start = [&](auto kernel, size_t smem, auto... args) {
    if (early)
      launch_early(kernel, grid, ATTN_WARPS * 32, smem, stream, args...);
    else
      kernel<<<grid, ATTN_WARPS * 32, smem, stream>>>(args...);
  };
  CUtensorMap tk, tv;
  const int pages = context > 0 ? (context + 127) / 128 + 1 : max_pages;
  if (attn_digits(D, rep, pages, splits, wide, kc, vc) && kv_map<D>(&tk, kc, kvh) &&
      kv_map<D>(&tv, vc, kvh)) {
    constexpr int D_ = D == 256 ? 128 : D;         // (256 channels: never)
    auto kernel = apart ? attn_digits_kernel<D_, true> : attn_digits_kernel<D_, false>;
    static const int slot[2] = {runtime_new_slot(), runtime_new_slot()};
    constexpr int SMEM = DigitTile<D_>::SMEM;
    if (const int e = runtime_allow_smem(slot[apart], kernel, SMEM)) return e;
    start(kernel, SMEM, tk, tv, q, gate, row_req, row_pos, page_table, max_pages, ks, vs, out, qh,
          kvh, splits, scratch, rep, apart_keys, runtime_status_ptr());
  } else {
    auto kernel =
        wide ? (apart ? attn_rows_kernel<D, true, true> : attn_rows_kernel<D, true, false>)
             : (apart ? attn_rows_kernel<D, false, true> : attn_rows_kernel<D, false, false>);
    static const int slot[4] = {runtime_new_slot(), runtime_new_slot(), runtime_new_slot(),
                                runtime_new_slot()};
    constexpr int SMEM = AttnTile<D>::SMEM;
    if (const int e = runtime_allow_smem(slot[2 * apart + wide], kernel, SMEM)) return e;
    start(kernel, SMEM, q, gate, row_req, row_pos, page_table, max_pages, kc, vc, ks, vs, out, qh,
          kvh, splits, scratch, rep, apart_keys);
  }
  if (splits > 1)
    launch_early(attn_merge_kernel<D>, dim3(rows, qh), D < 128 ? 64 : 128, 0, stream, scratch, gate,
                 out, qh, splits);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace orinfer

using namespace orinfer;

extern "C" size_t orinfer_attention_scratch_bytes(int rows, int qh, int head_dim, int splits) {
  if (splits <= 1) return 0;
  return static_cast<size_t>(rows) * qh * splits * (head_dim + 2) * sizeof(float);
}

// Whether the row kernel of such a call may start ahead of the end of the kernel in front.
extern "C" int orinfer_attention_starts_early(int rows, int kvh, int head_dim, int splits) {
  return attn_starts_early(head_dim, static_cast<long long>(rows) * kvh * splits) ? 1 : 0;
}

// Whether such a call takes the digit form (given aligned tensors).
extern "C" int orinfer_attention_in_digits(int qh, int kvh, int head_dim, int max_pages,
                                           int splits) {
  if (kvh <= 0 || qh % kvh || splits < 1) return 0;
  return attn_digits(head_dim, qh / kvh, max_pages, splits, true, nullptr, nullptr) ? 1 : 0;
}

extern "C" int orinfer_attention(const __half* q, const __half* gate, const int* row_req,
                                 const int* row_pos, const int* page_table, int max_pages,
                                 const int8_t* kc, const int8_t* vc, const __half* ks,
                                 const __half* vs, __half* out, int rows, int qh, int kvh,
                                 int head_dim, int splits, float* scratch, int context,
                                 cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (splits < 1 || (splits > 1 && scratch == nullptr) || kvh <= 0 || qh % kvh) return -1;
  const int rep = qh / kvh;
#define CASE(DD)                                                                            \
  if (head_dim == DD)                                                                       \
    return launch_attn<DD>(q, gate, row_req, row_pos, page_table, max_pages, kc, vc, ks, vs, \
                           out, rows, qh, kvh, rep, splits, scratch, context, stream);
  // query heads per KV head: the eight rows of a score tile (five only at D = 128)
  if (rep != 1 && rep != 2 && rep != 4 && rep != 8 && !(rep == 5 && head_dim == 128)) return -1;
  CASE(64) CASE(128) CASE(256)
#undef CASE
  return -1;
}
