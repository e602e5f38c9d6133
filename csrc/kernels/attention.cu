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

// One CTA per row and head.  The records' maxima and sums are read by a lane each and handed round,
// the outputs eight records at a time, since a call of few rows waits for each load in turn: with a
// record per step of the loop, and attn_finish computing every factor anew for each channel, one row
// of 2000 keys and 32 / 8 heads of 128 took 10.7 us (now 8.3), 16 / 2 heads of 256 (32 records) 15.1
// (10.0), 64 rows of 640 keys unsplit 26.8 (22.9).
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

template <int D>
static int launch_attn(const __half* q, const __half* gate, const int* row_req, const int* row_pos,
                       const int* page_table, int max_pages, const int8_t* kc, const int8_t* vc,
                       const __half* ks, const __half* vs, __half* out, int rows, int qh, int kvh,
                       int rep, int splits, float* scratch, cudaStream_t stream) {
  dim3 grid(rows, kvh, splits);
  const bool wide = ((reinterpret_cast<uintptr_t>(q) & 15) | (reinterpret_cast<uintptr_t>(ks) & 7) |
                     (reinterpret_cast<uintptr_t>(vs) & 7)) == 0;
  constexpr int SMEM = AttnTile<D>::SMEM;
  const long long ctas = splits > 1 || kvh < ATTN_WARPS ? 0 : static_cast<long long>(rows) * kvh;
  const long long waves = ctas / (148 * AttnTile<D>::MIN_CTAS);
  const int apart_keys = AttnTile<D>::KB * static_cast<int>(waves < 4 ? waves : 4);
  const bool apart = apart_keys > 0;
  auto kernel =
      wide ? (apart ? attn_rows_kernel<D, true, true> : attn_rows_kernel<D, true, false>)
           : (apart ? attn_rows_kernel<D, false, true> : attn_rows_kernel<D, false, false>);
  if (runtime_ensure_init() != cudaSuccess) return -2;
  static const int slot[4] = {runtime_new_slot(), runtime_new_slot(), runtime_new_slot(),
                              runtime_new_slot()};
  if (const int e = runtime_allow_smem(slot[2 * apart + wide], kernel, SMEM)) return e;
  if (attn_starts_early(D, static_cast<long long>(rows) * kvh * splits))
    launch_early(kernel, grid, ATTN_WARPS * 32, SMEM, stream, q, gate, row_req, row_pos, page_table,
                 max_pages, kc, vc, ks, vs, out, qh, kvh, splits, scratch, rep, apart_keys);
  else
    kernel<<<grid, ATTN_WARPS * 32, SMEM, stream>>>(q, gate, row_req, row_pos, page_table,
                                                    max_pages, kc, vc, ks, vs, out, qh, kvh,
                                                    splits, scratch, rep, apart_keys);
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

extern "C" int orinfer_attention(const __half* q, const __half* gate, const int* row_req,
                                 const int* row_pos, const int* page_table, int max_pages,
                                 const int8_t* kc, const int8_t* vc, const __half* ks,
                                 const __half* vs, __half* out, int rows, int qh, int kvh,
                                 int head_dim, int splits, float* scratch, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (splits < 1 || (splits > 1 && scratch == nullptr) || kvh <= 0 || qh % kvh) return -1;
  const int rep = qh / kvh;
#define CASE(DD)                                                                            \
  if (head_dim == DD)                                                                       \
    return launch_attn<DD>(q, gate, row_req, row_pos, page_table, max_pages, kc, vc, ks, vs, \
                           out, rows, qh, kvh, rep, splits, scratch, stream);
  // query heads per KV head: the eight rows of a score tile (five only at D = 128)
  if (rep != 1 && rep != 2 && rep != 4 && rep != 8 && !(rep == 5 && head_dim == 128)) return -1;
  CASE(64) CASE(128) CASE(256)
#undef CASE
  return -1;
}
