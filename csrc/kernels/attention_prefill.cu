// Causal GQA flash attention for prefill chunks over the paged INT8 KV cache, on tcgen05 tensor
// cores with TMEM accumulators.
//
// A query tile is 128 rows: P = 128 / rep consecutive query positions of one request times the
// `rep` query heads that share one KV head (the heads are packed into the MMA M axis so each INT8
// K/V page is dequantised once for all of them).  One CTA owns NQ tiles: in large packets of head
// sizes 64 and 128 two neighbouring ones, so that a dequantised page serves 256 rows and the
// tensor core works on one tile while the softmax warps of the other are busy.  Per step of KT
// keys:
//   * eight warps read the INT8 page and its group-64 FP16 scales straight from global memory (a
//     step ahead, in registers), dequantise to FP16 and store K and V as 128-byte-swizzled tiles
//     (K is the K-major B operand of S = Q K^T, V the MN-major B operand of O += P V);
//   * warp 1 issues tcgen05.mma kind::f16: S (128 x KT fp32) and O (128 x D fp32) live in TMEM;
//   * eight warps per tile own two threads per query row, each with half of the step's keys: they
//     read S from TMEM, apply scale and the causal mask, and write P as FP16 over their half of S,
//     where the second MMA reads it as its A operand.  The two meet once per step, for the row's
//     maximum, and hand over the sum of the weights, which are added in the order of the keys
//     (sums of their own per half would save 5 % of 4096 rows and 4 to 9 % of short chunks, and
//     move FP16 outputs by a step, which the INT8 rows of the next projection make a code step). P
//     is relative to the row's running maximum, so its largest weight is exactly 1 and O is
//     rescaled whenever a row of the warp finds a larger score;
//   * warp 0 loads the Q tiles once with a 3-D TMA (d, head, position).
// With one tile S is double buffered instead.  Head size 256 has room for no more (Q 64 KB, two K
// and two V buffers of 32 KB; TMEM: two S of 64 columns and O of 256) and walks the cache in half
// pages. CTAs are ordered from the last query positions (the longest walks) to the first.
//
// A step of two tiles is a chain per tile (softmax, P V, Q K^T of the next step) and two of them
// hide each other only in part: 5500 cycles for 128 keys with one softmax thread per row and the
// MMAs issued inside a branch on the lane, about 4700 with two threads and a whole warp in the
// issuing loop.  The tensor core needs 2050 of them, the exponentials as many. One 4096-token
// chunk, 32 / 8 heads of 128: 377 us with one tile per CTA and P in shared memory, 243 with two
// tiles and P in TMEM, 203 with two threads per row and a whole issuing warp (677 TFLOP/s causal);
// 512 tokens 19 -> 14 us, 64 behind 1000 29 -> 22.  A reference that follows the maximum only when
// it lags by 2^8 saves another tenth (fewer rescales of O) but rounds the largest weights in FP16:
// the error against 64 bits grows by 1.8 % there and by 3.7 % for 500 rows behind 1000.  Chunks of
// 777 and 646 rows behind 3000 positions, 16 / 2 gated heads of 256: 354 -> 276 -> 244 with K and
// V freed apart, 223 with plain loads, 161 with the gates asked for ahead (one at a time, two
// bytes of a row per lane, a tile's epilogue took 30 us; 17 rows 41 -> 10 us).
// Where the tiles are fewer than half the SMs, the CTAs of a cluster cut the keys of each (SPLIT):
// 64 rows behind 1000 positions 32 -> 18.5 us, 500 behind 1000 44 -> 32.5, 64 behind 20000 450 ->
// 72.  Heads of 64 and 128 channels are left whole: a step serves twice as many keys, so that a
// walk is half as long, and their FP16 outputs would move by a step here and there, which the INT8
// rows of the next projection make a code step (what the split would save there was not measured).
// Output is O / sum, optionally times sigmoid(gate), in FP16.  Replaces the prefill
// configurations of causal_attention_int8 and dequantize_attention_kv
// (kernels/cuda/model/attention_rows.py:61-276, kernels/cuda/model/kv_int8.py:210-247).
#include <cuda.h>

#include "api.h"
#include "common.cuh"
#include "tma.h"

namespace orinfer {
namespace fa {

constexpr int TILE = 128;                    // query rows per tile
constexpr int DQ_WARPS = 8;                  // dequantisation warps

template <int D, int NQ>                                 // NQ: query tiles per CTA
struct Smem {
  static constexpr int THREADS = (2 + 8 * NQ + DQ_WARPS) * 32;
  static constexpr int KT = D > 128 ? 64 : 128;          // keys per step
  static constexpr int SUB = TILE * 128;                 // one [128 x 64 fp16] sub-tile (Q)
  static constexpr int KSUB = KT * 128;                  // one [KT x 64 fp16] sub-tile (K, V)
  static constexpr int NSUB = D / 64;                    // sub-tiles per operand
  static constexpr int Q_OFF = 0;                        // NQ tiles
  static constexpr int K_OFF = Q_OFF + NQ * NSUB * SUB;  // two K buffers
  static constexpr int V_OFF = K_OFF + 2 * NSUB * KSUB;  // two V buffers
  static constexpr int BAR_OFF = V_OFF + 2 * NSUB * KSUB;
  static constexpr int MAX_OFF = BAR_OFF + 256;          // [NQ][2 steps][2 halves][128] row maxima
  static constexpr int SUM_OFF = MAX_OFF + NQ * 4 * TILE * 4;   // [NQ][128] sums of first halves
  static constexpr int PAIR_OFF = SUM_OFF + NQ * TILE * 4;      // [NQ][QUADS][128], see `pair`
  static constexpr int QUADS = KT == 64 ? 0 : D == 128 && NQ == 2 ? 7 : 8;
  static constexpr int TOTAL = PAIR_OFF + NQ * QUADS * TILE * 16 + 1024;
  static_assert(TOTAL <= 227 * 1024, "exceeds the shared memory of one CTA");
};

__device__ __forceinline__ void mma_f16_ss_by(uint32_t leader, uint32_t tmem_d, uint64_t adesc,
                                              uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A holds two FP16 values of a row per 32-bit column.
__device__ __forceinline__ void mma_f16_ts_by(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a,
                                              uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Eight INT8 values (two words) -> eight FP16 values times an FP16 scale, exactly
// half(float(q) * float(scale)): build 1152 + q as a half via byte permute, subtract,
// multiply (one rounding, like the fp32 product rounded to half).
__device__ __forceinline__ uint4 dequant8(uint32_t w0, uint32_t w1, __half2 scale2) {
  const __half2 bias = __half2half2(__ushort_as_half(0x6480));     // 1152.0
  uint32_t x0 = w0 ^ 0x80808080u, x1 = w1 ^ 0x80808080u;
  uint32_t h[4];
  h[0] = __byte_perm(x0, 0x64646464u, 0x4140);
  h[1] = __byte_perm(x0, 0x64646464u, 0x4342);
  h[2] = __byte_perm(x1, 0x64646464u, 0x4140);
  h[3] = __byte_perm(x1, 0x64646464u, 0x4342);
  uint4 out;
  uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __half2 v = *reinterpret_cast<__half2*>(&h[i]);
    v = __hmul2(__hsub2(v, bias), scale2);
    o[i] = *reinterpret_cast<uint32_t*>(&v);
  }
  return out;
}

// The gates of 32 channels of an output row (a row of its own per lane, so each load waits for a
// line of its own: they are asked for well ahead of their use).
struct Gates {
  uint4 w[4];
  __device__ __forceinline__ void load(const __half* gate, size_t at) {
    if ((reinterpret_cast<uintptr_t>(gate) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = reinterpret_cast<const uint4*>(gate + at)[i];
    } else {
      __half* h = reinterpret_cast<__half*>(w);
#pragma unroll
      for (int i = 0; i < 32; ++i) h[i] = gate[at + i];
    }
  }
};
// Eight channels of an output row, times the sigmoids of their gates.
__device__ __forceinline__ void store_gated(float (&v)[8], bool gated, const uint4& gates,
                                            __half* out) {
  __align__(16) __half h[8];
  if (gated) {
    const __half2* g = reinterpret_cast<const __half2*>(&gates);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 sg = sigmoid_pair(__half22float2(g[i]));
      v[2 * i] *= sg.x;
      v[2 * i + 1] *= sg.y;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) h[i] = __float2half_rn(v[i]);
  *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(h);
}

struct Chunk {            // one prefill chunk of one request
  int row_start;          // first packed row
  int q_len;              // rows in the chunk
  int pos0;               // absolute position of the first row
  int slot;               // row of the page table
};

// SPLIT (one tile per CTA): the CTAs of a cluster take the tile's keys in equal parts, and each
// then puts one slice of the channels together from everybody's shared memory.
__device__ __forceinline__ float4 cluster_float4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ float cluster_float(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
constexpr int SPLIT_STEPS = 3;               // a part has at least as many steps

template <int D, int NQ, bool GATED, bool SPLIT>
__global__ void __launch_bounds__(Smem<D, NQ>::THREADS, 1) attn_prefill_kernel(
    const __grid_constant__ CUtensorMap tmap_q, const Chunk* chunks, const int* page_table,
    int max_pages, const int8_t* kc, const int8_t* vc, const __half* ks, const __half* vs,
    const __half* gate, __half* __restrict__ out, int qh, int kvh, int rep, int num_pages,
    int ranks, int* status) {
  static_assert(!SPLIT || NQ == 1, "a split tile has its CTA to itself");
  using L = Smem<D, NQ>;
  constexpr int NSUB = L::NSUB, KT = L::KT;
  constexpr int GROUPS = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr int S_STRIDE = KT;                    // S of tile q (NQ = 2) or of buffer b (NQ = 1)
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* q_full = bars;            // Q tiles landed
  uint64_t* k_ready = bars + 1;       // [2] dequantised K buffer filled
  uint64_t* v_ready = bars + 3;       // [2] dequantised V buffer filled
  uint64_t* s_full = bars + 5;        // [2] S = QK^T finished (per tile, or per buffer)
  uint64_t* p_ready = bars + 7;       // [2] P written over S, O rescaled (an arrival per warp)
  uint64_t* o_done = bars + 9;        // [2] O += PV finished (per tile)
  uint64_t* k_free = bars + 11;       // [2] the last MMA that read K buffer b finished
  uint64_t* v_free = bars + 13;       // [2] the same for V
  uint64_t* sum_ready = bars + 15;    // [NQ][4] sums of the first halves of 32 rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15 + 4 * NQ);

  const int warp = warp_same(threadIdx.x >> 5), lane = threadIdx.x & 31;
  grid_wait();
  const Chunk ch = chunks[blockIdx.z];
  const int h = blockIdx.y;                       // kv head
  const int P = TILE / rep;                       // query positions per tile
  // first chunk-relative position of this CTA's tiles; long walks start first
  const int rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = SPLIT ? blockIdx.x / ranks : blockIdx.x;
  const int tiles = SPLIT ? gridDim.x / ranks : gridDim.x;
  const int p_first = (tiles - 1 - tile) * NQ * P;
  if (p_first >= ch.q_len) return;
  // steps that any row of tile q can see (0: the chunk ends before the tile)
  auto steps_of = [&](int q) {
    const int first = p_first + q * P;
    return first >= ch.q_len ? 0 : (ch.pos0 + min(first + P, ch.q_len) - 1) / KT + 1;
  };
  const int kv_end = ch.pos0 + min(p_first + NQ * P, ch.q_len);
  int n_steps[NQ], n_max = 0;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    n_steps[q] = steps_of(q);
    n_max = max(n_max, n_steps[q]);
  }
  int j0 = 0;                                     // this CTA's first step; others count from it
  if (SPLIT) {
    const int parts = max(1, min(ranks, n_max / SPLIT_STEPS));
    j0 = rank < parts ? n_max * rank / parts : 0;
    n_max = rank < parts ? n_max * (rank + 1) / parts - j0 : 0;
    n_steps[0] = n_max;
  }

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&k_ready[b], DQ_WARPS);
      mbar_init(&v_ready[b], DQ_WARPS);
      mbar_init(&s_full[b], 1);
      mbar_init(&p_ready[b], 8);
      mbar_init(&o_done[b], 1);
      mbar_init(&k_free[b], 1);
      mbar_init(&v_free[b], 1);
    }
    for (int b = 0; b < 4 * NQ; ++b) mbar_init(&sum_ready[b], 1);
    mbar_fence_init();
    prefetch_tmap(&tmap_q);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_same(*tmem_slot);
  grid_release();
  const uint32_t tmem_s = tmem_base, tmem_o = tmem_base + 256;   // O of tile q at + q * 128
  const int* pages = page_table + static_cast<size_t>(ch.slot) * max_pages;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, static_cast<uint32_t>(NQ) * NSUB * 64 * 2 * rep * P);
      for (int q = 0; q < NQ; ++q)
        for (int s = 0; s < NSUB; ++s)
          tma_load_3d(smem + L::Q_OFF + (q * NSUB + s) * L::SUB, &tmap_q, q_full, s * 64, h * rep,
                      ch.row_start + p_first + q * P);
      mbar_wait(q_full, 0, status, STATUS_TMA_WAIT, 1);     // our copies have landed before exit
    }
  } else if (warp == 1) {
    // the whole warp runs the loop (see elect_one)
    constexpr uint32_t idesc_s = umma_idesc(1, 0, 0, 0, 0, TILE, KT);
    constexpr uint32_t idesc_o = umma_idesc(1, 0, 0, 0, 1, TILE, D);
    const uint32_t leader = elect_one();
    const uint64_t qd = umma_desc(smem_u32(smem + L::Q_OFF), 16, 1024);
    const uint64_t kd = umma_desc(smem_u32(smem + L::K_OFF), 16, 1024);
    const uint64_t vd = umma_desc(smem_u32(smem + L::V_OFF), L::KSUB, 1024);
    int steps[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) steps[q] = warp_same(n_steps[q]);
    const int last = warp_same(n_max);
    bool ok = __all_sync(0xffffffffu, mbar_wait(q_full, 0, status, STATUS_MMA_WAIT, 2));
    auto wait_for = [&](uint64_t* bar, uint32_t parity, int detail) {
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, status, STATUS_MMA_WAIT, detail));
      tc_fence_after();
    };
    auto issue_qk = [&](int q, int j) {
      const int sb = NQ == 2 ? q : j & 1;
      const uint64_t kb = kd + static_cast<uint64_t>((j & 1) * NSUB * L::KSUB / 16);
#pragma unroll
      for (int i = 0; i < D / 16; ++i)
        mma_f16_ss_by(leader, tmem_s + S_STRIDE * sb,
                      qd + ((q * NSUB + i / 4) * L::SUB + i % 4 * 32) / 16,
                      kb + (i / 4 * L::KSUB + i % 4 * 32) / 16, idesc_s, i != 0 ? 1u : 0u);
      tc_commit_by(leader, &s_full[sb]);
    };
    auto issue_pv = [&](int q, int j) {
      const int sb = NQ == 2 ? q : j & 1;
      wait_for(&p_ready[sb], (NQ == 2 ? j : j >> 1) & 1, 0x200 | (j & 0xff));
      if (!ok) return;
      const uint64_t vb = vd + static_cast<uint64_t>((j & 1) * NSUB * L::KSUB / 16);
#pragma unroll
      for (int i = 0; i < KT / 16; ++i)
        mma_f16_ts_by(leader, tmem_o + 128 * q,
                      tmem_s + S_STRIDE * sb + i / (KT / 32) * (KT / 2) + i % (KT / 32) * 8,
                      vb + i * 2048 / 16, idesc_o, (j | i) != 0 ? 1u : 0u);
      tc_commit_by(leader, &o_done[q]);
    };
    // MMAs of one thread run in order.  NQ = 2: QK of step j + 1 overwrites the P of step j of
    // the same tile, so it follows that tile's PV; meanwhile the other tile's softmax runs.
    // NQ = 1: QK of step j + 1 goes into the other S buffer, ahead of PV of step j.
    auto next_qk = [&](int q, int j) {                // tile q's part of QK of step j
      if (q == 0) wait_for(&k_ready[j & 1], (j >> 1) & 1, 0x100 | (j & 0xff));
      if (ok && j < steps[q]) issue_qk(q, j);
      if (ok && q == NQ - 1) tc_commit_by(leader, &k_free[j & 1]);
    };
    if (!SPLIT || last > 0) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) next_qk(q, 0);
    }
    for (int j = 0; j < last && ok; ++j) {
      const bool more = j + 1 < last;
      if (NQ == 1 && more) next_qk(0, j + 1);
      wait_for(&v_ready[j & 1], (j >> 1) & 1, 0x180 | (j & 0x7f));
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        if (ok && j < steps[q]) issue_pv(q, j);
        if (q == NQ - 1 && ok) tc_commit_by(leader, &v_free[j & 1]);
        if (NQ == 2 && ok && more) next_qk(q, j + 1);
      }
    }
    __syncwarp();
  } else if (warp >= 2 + 8 * NQ) {
    // ---------------- dequant warps: INT8 page -> FP16 swizzled K / V tiles
    // The raw rows of step j + 1 are in flight while step j is multiplied.  K and V have two
    // buffers each, freed apart.  With one tile K of step j + 1 is converted while PV of step j - 1
    // still reads V, so that the next Q K^T does not wait for it (777 and 646 rows behind 3000, 16
    // / 2 heads of 256: 276 -> 244 us; 512 rows, 32 / 8 heads of 128: 15.3 -> 14.6).  With two
    // tiles that wait is hidden, and the conversions do better in one piece (4096 rows 216 us, 219
    // apart).
    constexpr int CPK = D / 16;                      // 16-byte chunks per key
    constexpr int DQ = DQ_WARPS * 32, ITERS = KT * CPK / DQ;
    uint4 kraw[ITERS], vraw[ITERS];
    __half ksc[ITERS], vsc[ITERS];
    const int u = threadIdx.x - (2 + 8 * NQ) * 32;
    const int rows = (DQ / CPK) * kvh;               // the rows of a thread are that far apart
    auto load = [&](int j, int page, bool k, bool v) {
      // one base address per step
      const size_t slot =
          (static_cast<size_t>(page) * 128 + (j0 + j) * KT % TILE + u / CPK) * kvh + h;
      const int8_t* kp = kc + slot * D + (u % CPK) * 16;
      const int8_t* vp = vc + slot * D + (u % CPK) * 16;
      const __half* ksp = ks + slot * GROUPS + (u % CPK) / 4;
      const __half* vsp = vs + slot * GROUPS + (u % CPK) / 4;
      // Keys past the last position that a row of this CTA sees may be slots never written.  Their
      // weight is zero, but zero times an infinite or NaN value is not: they get no value scale.
      const int live = kv_end - (j0 + j) * KT - u / CPK;
#pragma unroll
      for (int it = 0; it < ITERS; ++it) {
        const size_t at = static_cast<size_t>(it) * rows;
        if (k) {
          kraw[it] = *reinterpret_cast<const uint4*>(kp + at * D);
          ksc[it] = ksp[at * GROUPS];
        }
        if (v) {
          vraw[it] = *reinterpret_cast<const uint4*>(vp + at * D);
          vsc[it] = it * (DQ / CPK) < live ? vsp[at * GROUPS] : __half(0.f);
        }
      }
    };
    auto place = [&](unsigned char* to, const uint4& raw, __half sc, int it) {
      const int key = it * (DQ / CPK) + u / CPK, c = u % CPK, chunk = (c % 4) * 2;
      const __half2 s2 = __half2half2(sc);
      unsigned char* dst = to + (c / 4) * L::KSUB;
      *reinterpret_cast<uint4*>(dst + swz128(key, chunk)) = dequant8(raw.x, raw.y, s2);
      *reinterpret_cast<uint4*>(dst + swz128(key, chunk + 1)) = dequant8(raw.z, raw.w, s2);
    };
    auto convert = [&](int buf, bool k, bool v) {
#pragma unroll
      for (int it = 0; it < ITERS; ++it) {
        if (k) place(smem + L::K_OFF + buf * NSUB * L::KSUB, kraw[it], ksc[it], it);
        if (v) place(smem + L::V_OFF + buf * NSUB * L::KSUB, vraw[it], vsc[it], it);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && k) mbar_arrive(&k_ready[buf]);
      if (lane == 0 && v) mbar_arrive(&v_ready[buf]);
    };
    auto page_of = [&](int j) {
      const int page = pages[(j0 + j) * KT / TILE];
      if (page >= 0 && page < num_pages) return page;
      report_status(status, STATUS_BAD_INDEX, 3);
      return 0;
    };
    bool ok = true;
    int page = 0;
    if (!SPLIT || n_max > 0) {
      page = page_of(0);
      load(0, page, true, true);
    }
    if (n_max > 1) page = page_of(1);
    // a buffer was last read by the MMAs of step j - 2
    auto released = [&](uint64_t* free, int j) {
      if (j >= 2)
        ok = ok && mbar_wait(&free[j & 1], ((j >> 1) - 1) & 1, status, STATUS_DECODE_WAIT, j);
      ok = __all_sync(0xffffffffu, ok);
    };
    for (int j = 0; j < n_max; ++j) {
      const int buf = j & 1;
      released(k_free, j);
      if (NQ == 1) {
        if (!ok) break;
        convert(buf, true, false);
        if (j + 1 < n_max) load(j + 1, page, true, false);
      }
      released(v_free, j);
      if (!ok) break;
      convert(buf, NQ == 2, true);
      if (j + 1 < n_max) load(j + 1, page, NQ == 2, true);
      if (j + 2 < n_max) page = page_of(j + 2);
    }
  } else {
    // ---------------- softmax warps: two threads per query row, each with half of a step's keys
    const int q = (warp - 2) >> 3;                          // tile
    const int half = ((warp - 2) >> 2) & 1;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;                       // row of the tile = TMEM lane
    const int first = p_first + q * P;
    const int p_rel = row / rep, head = h * rep + row % rep;
    const bool valid = row < P * rep && first + p_rel < ch.q_len;
    const int q_pos = valid ? ch.pos0 + first + p_rel : -1;
    const float scale = rsqrtf(static_cast<float>(D)) * 1.4426950408889634f;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    constexpr int KH = KT / 2, DH = D / 2;                  // keys and channels of a thread
    const uint32_t tmem_oq = tmem_o + 128 * q + half * DH + lane_addr;
    const int steps = NQ == 2 && q == 1 ? n_steps[NQ - 1] : n_steps[0];
    // maxima of both halves, double buffered: a slot is rewritten two exchanges later
    float* row_max = reinterpret_cast<float*>(smem + L::MAX_OFF) + q * 4 * TILE + row;
    auto meet = [&]() {                                     // the two warps of these rows
      asm volatile("bar.sync %0, 64;" ::"r"(1 + q * 4 + quad) : "memory");
    };
    // A row's weights are added up in the order of its keys: the thread of the second half goes on
    // where that of the first one ended.  It does so when P is on its way; until then it keeps the
    // sums of two weights, four to a quad, in registers or (two tiles) most of them in shared
    // memory.
    float* first_sum = reinterpret_cast<float*>(smem + L::SUM_OFF) + q * TILE + row;
    float4* quads = reinterpret_cast<float4*>(smem + L::PAIR_OFF) + q * L::QUADS * TILE + row;
    uint64_t* handed = &sum_ready[q * 4 + quad];
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < steps; ++j) {
      const int sb = NQ == 2 ? q : j & 1;
      const uint32_t parity = (NQ == 2 ? j : j >> 1) & 1;
      const uint32_t tmem_sj = tmem_s + S_STRIDE * sb + half * KH + lane_addr;
      ok = ok && mbar_wait(&s_full[sb], parity, status, STATUS_EPILOGUE_WAIT, j);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {                                  // a warp that gave up still meets its partner
        meet();
        continue;
      }
      tc_fence_after();
      const int key0 = (j0 + j) * KT + half * KH;
      // Only the last page of a row can hold keys beyond its position; every earlier page
      // takes the mask-free path.
      const bool full_warp = __all_sync(0xffffffffu, key0 + KH - 1 <= q_pos);
      // pass 1: row maximum (of the raw scores: the scale is positive); the first 32 scores stay in
      // registers
      uint32_t r[32];
      float m0 = -INFINITY, m1 = -INFINITY;
      auto peak = [&](int c0) {
        tmem_ld_32x32(tmem_sj + c0, r);
        tc_wait_ld();
        if (full_warp) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            m0 = fmaxf(m0, __uint_as_float(r[i]));
            m1 = fmaxf(m1, __uint_as_float(r[i + 1]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + c0 + i <= q_pos) m0 = fmaxf(m0, __uint_as_float(r[i]));
        }
      };
      if (KH == 64) peak(32);
      peak(0);
      float* slot = row_max + (j & 1) * 2 * TILE;
      slot[half * TILE] = fmaxf(m0, m1);
      meet();
      const float m_tile = fmaxf(slot[0], slot[TILE]) * scale;      // -inf stays -inf
      const float m_new = fmaxf(m_run, m_tile);
      const float corr = m_new == -INFINITY ? 1.f : ex2(m_run - m_new);
      // pass 2: probabilities -> FP16 over the scores already read; their sum, or its terms
      float l_tile = 0.f;
      float4 kept[KH / 8 > L::QUADS ? KH / 8 - L::QUADS : 1];
      auto quad_of = [&](int i) -> float4& {
        return i < L::QUADS ? quads[i * TILE] : kept[i < L::QUADS ? 0 : i - L::QUADS];
      };
      auto weigh = [&](int c0) {
        uint32_t packed[16];
        float pair[16];
        if (full_warp) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = ex2(fmaf(__uint_as_float(r[i]), scale, -m_new));
            const float p1 = ex2(fmaf(__uint_as_float(r[i + 1]), scale, -m_new));
            pair[i / 2] = p0 + p1;
            const __half2 hp = __floats2half2_rn(p0, p1);
            packed[i / 2] = *reinterpret_cast<const uint32_t*>(&hp);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0 = ex2(fmaf(__uint_as_float(r[i]), scale, -m_new));
            float p1 = ex2(fmaf(__uint_as_float(r[i + 1]), scale, -m_new));
            if (key0 + c0 + i > q_pos) p0 = 0.f;
            if (key0 + c0 + i + 1 > q_pos) p1 = 0.f;
            pair[i / 2] = p0 + p1;
            const __half2 hp = __floats2half2_rn(p0, p1);
            packed[i / 2] = *reinterpret_cast<const uint32_t*>(&hp);
          }
        }
        tmem_st_32x16(tmem_sj + c0 / 2, packed);
        if (half == 0) {
#pragma unroll
          for (int i = 0; i < 16; ++i) l_tile += pair[i];
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            quad_of((c0 + 2 * i) / 8) = make_float4(pair[i], pair[i + 1], pair[i + 2], pair[i + 3]);
        }
      };
      weigh(0);
      if (KH == 64) {
        tmem_ld_32x32(tmem_sj + 32, r);
        tc_wait_ld();
        weigh(32);
      }
      if (half == 0) {
        *first_sum = l_tile;
        __syncwarp();
        if (lane == 0) mbar_arrive(handed);
      }
      // O holds steps 0..j-1 once PV of step j-1 is done.  Waited for at every step, so that no
      // wait is ever two phases away from its barrier; NQ = 2: it is done, QK ran after it.
      if (j >= 1) {
        ok = mbar_wait(&o_done[q], (j - 1) & 1, status, STATUS_EPILOGUE_WAIT, 0x100 | j);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) continue;
        tc_fence_after();
      }
      if (j >= 1 && !__all_sync(0xffffffffu, corr == 1.f)) {
#pragma unroll 1
        for (int c0 = 0; c0 < DH; c0 += 32) {
          tmem_ld_32x32(tmem_oq + c0, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
          tmem_st_32x32(tmem_oq + c0, r);
        }
      }
      tc_wait_st();
      m_run = m_new;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[sb]);
      if (half == 1) {
        ok = mbar_wait(handed, j & 1, status, STATUS_EPILOGUE_WAIT, 0x200 | j);
        ok = __all_sync(0xffffffffu, ok);
        l_tile = *first_sum;
#pragma unroll
        for (int i = 0; i < KH / 8; ++i) {
          const float4 v = quad_of(i);
          l_tile = (((l_tile + v.x) + v.y) + v.z) + v.w;
        }
        l_run = l_run * corr + l_tile;
      }
    }
    const bool gated = GATED && !SPLIT && valid;
    const size_t orow = static_cast<size_t>(ch.row_start + first + p_rel) * qh + head;
    Gates ahead;
    if (gated) ahead.load(gate, orow * D + half * DH);
    if (ok && steps > 0) {
      ok = mbar_wait(&o_done[q], (steps - 1) & 1, status, STATUS_EPILOGUE_WAIT, 0x300);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (half == 1) *first_sum = l_run;
    meet();
    if (SPLIT) {
      // this part's O, four channels of all rows at a time, where K and V were; its maximum and sum
      tc_fence_after();
      float* stat = reinterpret_cast<float*>(smem + L::MAX_OFF);
      if (half == 0) {
        stat[row] = ok && steps > 0 ? m_run : -INFINITY;
        stat[TILE + row] = *first_sum;
      }
      float4* part = reinterpret_cast<float4*>(smem + L::K_OFF);
      if (ok && steps > 0) {
#pragma unroll 1
        for (int c0 = 0; c0 < DH; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tmem_oq + c0, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            part[(half * DH + c0 + i) / 4 * TILE + row] =
                make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]),
                            __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
        }
      }
    } else if (ok && steps > 0) {
      tc_fence_after();
      const float l_all = *first_sum;
      const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
#pragma unroll 1
      for (int c0 = 0; c0 < DH; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_oq + c0, r);
        const size_t at = orow * D + half * DH + c0;
        const Gates now = ahead;
        if (gated && c0 + 32 < DH) ahead.load(gate, at + 32);
        tc_wait_ld();
        if (valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[i + k]) * inv;
            store_gated(v, gated, now.w[i / 8], out + at + i);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
  if (SPLIT) {
    static_assert(!SPLIT || 4 * NSUB * L::KSUB >= D * TILE * 4, "O takes the place of K and V");
    cluster_sync_all();
    if (warp >= 2 && warp < 10) {
      const int half = ((warp - 2) >> 2) & 1, row = (warp & 3) * 32 + lane;
      const int p_rel = row / rep, head = h * rep + row % rep;
      const int slice = D / ranks / 2, c_lo = rank * 2 * slice + half * slice;   // channels
      if (row < P * rep && p_first + p_rel < ch.q_len) {
        const uint32_t stat = smem_u32(smem + L::MAX_OFF) + row * 4;
        const uint32_t part = smem_u32(smem + L::K_OFF) + (c_lo / 4 * TILE + row) * 16;
        float m = -INFINITY, l = 0.f;
        for (int s = 0; s < ranks; ++s) m = fmaxf(m, cluster_float(mapa_u32(stat, s)));
        float f[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          if (s >= ranks) break;
          const float ms = cluster_float(mapa_u32(stat, s));
          f[s] = ms == -INFINITY ? 0.f : ex2(ms - m);
          if (f[s] != 0.f) l = fmaf(cluster_float(mapa_u32(stat + TILE * 4, s)), f[s], l);
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const size_t at =
            (static_cast<size_t>(ch.row_start + p_first + p_rel) * qh + head) * D + c_lo;
#pragma unroll 1
        for (int c = 0; c < slice; c += 8) {
          float v[8];
          uint4 gates = make_uint4(0, 0, 0, 0);
          if (GATED) {
            if ((reinterpret_cast<uintptr_t>(gate) & 15) == 0) {
              gates = *reinterpret_cast<const uint4*>(gate + at + c);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) reinterpret_cast<__half*>(&gates)[i] = gate[at + c + i];
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = 0.f;
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            if (s >= ranks) break;
            if (f[s] == 0.f) continue;               // (nothing was put there)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const float4 o = cluster_float4(mapa_u32(part + (c / 4 + k) * TILE * 16, s));
              v[4 * k] = fmaf(o.x, f[s], v[4 * k]);
              v[4 * k + 1] = fmaf(o.y, f[s], v[4 * k + 1]);
              v[4 * k + 2] = fmaf(o.z, f[s], v[4 * k + 2]);
              v[4 * k + 3] = fmaf(o.w, f[s], v[4 * k + 3]);
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] *= inv;
          store_gated(v, GATED, gates, out + at + c);
        }
      }
    }
    __syncwarp();                                    // (the barrier wants whole warps)
    cluster_sync_all();                              // nobody leaves while its memory is read
  }
}

template <int D, int NQ, bool SPLIT = false>
int launch(const __half* q, const __half* gate, const Chunk* chunks, int n_chunks, int max_q_len,
           int total_rows, const int* page_table, int max_pages, const int8_t* kc,
           const int8_t* vc, const __half* ks, const __half* vs, __half* out, int qh, int kvh,
           int num_pages, cudaStream_t stream, int ranks = 1) {
  using L = Smem<D, NQ>;
  const int rep = qh / kvh;
  const int P = TILE / rep;
  PFN_encodeTiled enc = runtime_tma_encoder();
  if (!enc) return -3;
  CUtensorMap tq;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(qh),
                        static_cast<cuuint64_t>(total_rows)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(D) * 2, static_cast<cuuint64_t>(qh) * D * 2};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(rep), static_cast<cuuint32_t>(P)};
  cuuint32_t estr[3] = {1, 1, 1};
  if (enc(&tq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(q), dims, strides, box,
          estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return -3;
  static const int slot[2] = {runtime_new_slot(), runtime_new_slot()};
  auto kernel = gate ? attn_prefill_kernel<D, NQ, true, SPLIT>
                     : attn_prefill_kernel<D, NQ, false, SPLIT>;
  if (const int e = runtime_allow_smem(slot[gate != nullptr], kernel, L::TOTAL)) return e;
  dim3 grid((max_q_len + NQ * P - 1) / (NQ * P) * ranks, kvh, n_chunks);
  if (SPLIT) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = L::THREADS;
    cfg.dynamicSmemBytes = L::TOTAL;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tq, chunks, page_table, max_pages, kc,
                                             vc, ks, vs, gate, out, qh, kvh, rep, num_pages, ranks,
                                             runtime_status_ptr());
    return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
  }
  launch_early(kernel, grid, L::THREADS, L::TOTAL, stream, tq, chunks, page_table, max_pages, kc,
               vc, ks, vs, gate, out, qh, kvh, rep, num_pages, ranks, runtime_status_ptr());
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fa
}  // namespace orinfer

using namespace orinfer;

// Into how many parts the keys of a tile go (heads of 256 channels, one tile per CTA), the steps
// counted from the longest context, or where the caller does not know it from the page table's
// width: a serving engine's tables have the width of the longest context there may be, and 17 rows
// without a prefix are one step.  A step takes 1.35 us, a CTA about six of them besides, and a part
// five more to be put together with the others; a larger number has to save 15 %.  (More parts than
// SMs did not pay: 180 CTAs of 60 steps 161 us whole, 152 in two parts, 195 in four, but 188 of 12
// steps 45 and 72.)
static int prefill_ranks(long long ctas, long long steps) {
  int best = 1;
  double least = 0;
  for (int s = 1; s <= 8; s *= 2) {
    if (s > 1 && ctas * s > 148) break;
    const double waves = static_cast<double>((ctas * s + 147) / 148);
    const double cost = waves * (static_cast<double>(steps) / s + (s > 1 ? 11.0 : 6.0));
    if (s == 1 || cost < least * 0.85) {
      least = cost;
      best = s;
    }
  }
  return best;
}
extern "C" int orinfer_attention_prefill_parts(int ctas, int max_pages) {
  return prefill_ranks(ctas, static_cast<long long>(max_pages) * 2);
}

// chunks: int32 [n_chunks, 4] = (row_start, q_len, pos0, page-table row) on the device.
// context: positions that the chunks reach at most (pos0 + q_len), 0 where the caller cannot tell.
extern "C" int orinfer_attention_prefill(const __half* q, const __half* gate, const int* chunks,
                                         int n_chunks, int max_q_len, int total_rows,
                                         const int* page_table, int max_pages, const int8_t* kc,
                                         const int8_t* vc, const __half* ks, const __half* vs,
                                         __half* out, int qh, int kvh, int head_dim, int num_pages,
                                         int context, cudaStream_t stream) {
  if (n_chunks <= 0 || max_q_len <= 0) return 0;
  if (kvh <= 0 || qh % kvh || qh / kvh > 16) return -1;
  if (runtime_ensure_init() != cudaSuccess) return -2;
  const fa::Chunk* ch = reinterpret_cast<const fa::Chunk*>(chunks);
  // One tile per CTA while those CTAs fit about one wave: 512 rows of 32 / 8 heads of 128 17.7 us
  // against 21.8 with two (128 and 64 CTAs), 152 tiles 20.9 against 24.2; from 168 tiles on two
  // share their pages' conversion at no loss of width (28.4 against 25.4 us; 4096 rows 279 against
  // 241).  The longest chunk times their number overstates ragged packets, the rows in all and one
  // cut tile per chunk those that do not fill the buffer: the smaller of the two counts.
  const int tile_rows = fa::TILE / (qh / kvh);
  const long long longest =
      static_cast<long long>((max_q_len + tile_rows - 1) / tile_rows) * n_chunks;
  const long long packed = static_cast<long long>(total_rows / tile_rows) + n_chunks;
  const bool one = (longest < packed ? longest : packed) * kvh <= 160;
#define ORINFER_PREFILL(D, NQ)                                                                 \
  return fa::launch<D, NQ>(q, gate, ch, n_chunks, max_q_len, total_rows, page_table, max_pages, \
                           kc, vc, ks, vs, out, qh, kvh, num_pages, stream)
  if (head_dim == 128 && one) ORINFER_PREFILL(128, 1);
  if (head_dim == 128) ORINFER_PREFILL(128, 2);
  if (head_dim == 64 && one) ORINFER_PREFILL(64, 1);
  if (head_dim == 64) ORINFER_PREFILL(64, 2);
#undef ORINFER_PREFILL
  if (head_dim == 256) {
    const long long ctas = (longest < packed ? longest : packed) * kvh;
    const long long steps = static_cast<long long>(max_pages) * 2, known = (context + 63LL) / 64;
    const int ranks = prefill_ranks(ctas, context > 0 && known < steps ? known : steps);
    return (ranks > 1 ? fa::launch<256, 1, true> : fa::launch<256, 1, false>)(
        q, gate, ch, n_chunks, max_q_len, total_rows, page_table, max_pages, kc, vc, ks, vs, out,
        qh, kvh, num_pages, stream, ranks);
  }

  return -4;          // unsupported head size: caller falls back to the row kernel
}
