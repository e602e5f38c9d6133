// Quantised GEMM over many output tiles: one CTA per SM walks a list of (MT * 128) x 128 tiles,
// with every stage of the work in warps of its own.  The same product as qgemm_tc_kernel
// (gemm_tc.cu), bit for bit, for launches of more tiles than SMs: long prompts through wide
// projections and the grouped projections of mixture-of-experts layers
// (kernels/cuda/model/e8p_q4.py:144-265, kernels/cuda/model/integer_vq.py:263 and
// kernels/cuda/model/int8_projection.py:15 of the reference).
//
//   warp 0       activation tiles by TMA
//   warp 2       packed codes as bulk copies (INT8 weights: tiles by TMA)
//   warps 12..27 lattice codes -> INT8 weight tile
//   warp 1       tcgen05.mma kind::i8 into TMEM
//   warps 4..11  TMEM -> scales -> FP16 -> whole 64-byte pieces of rows
//
// A CTA of the one-tile kernel spends 33000 of 50000 cycles on 20 k-blocks of 512 x 128; the rest
// is its start (barriers, TMEM, tables: 1200), the first copies and the first decode (3000), its
// epilogue (9500) and the gap to the next CTA (2700), all of it with an idle tensor core.  Here the
// ring runs on across tiles, the epilogue has its own warps, and TMEM holds two sets of
// accumulators (MT = 1 or 2).
//
// What bounds it: INT8 weights take 67 cycles per 128 x 128 x 32 MMA when their copies are there
// (2048 x 19456 x 2560 126 -> 86 us, 2.4 PFLOP/s).  Lattice codes: the decode warps (67 % of the
// issue slots, the shared-memory pipe as busy, the tensor core 27 %).  With all sixteen on one
// k-block, each decoded for 540 to 650 of its 1280 to 1500 cycles; the rest were two waits (170
// each), the fence and the hand-overs.  So groups of them take k-blocks in turn, each warp with
// twice (Q2 with one row tile: four times) as many rows between two waits: 128 Q4 experts of 768, a
// whole layer, 2048 rows 292 -> 270 us, 1024 rows 243 -> 210, 300 rows 211 -> 179; 512 Q2 experts
// of 512, 2048 rows 619 -> 539, 1024 rows 519 -> 439 (Q4 in four groups: 223 where two take 214).
// Signs from arithmetic instead of lookups made a layer a sixth longer; codes loaded into registers
// from global memory four k-blocks ahead, with a 64 KB table whose addresses are single byte
// permutes (a quarter fewer instructions), 303 against 292 us: the loads are waited for.  The whole
// layer came from 447 us over 340 (this kernel) and 326 (the router's and the launches' share;
// votes on every wait and the activations' own barrier cost 1.5 %), and 15 us of 305 went with
// lookups that collide.
#include <cuda.h>

#include "api.h"
#include "common.cuh"
#include "gemm_walk.h"
#include "tma.h"

namespace orinfer {
namespace walk {

constexpr int BM = 128, BN = 128, BK = 128;
constexpr int TILE = 128 * 128;                    // bytes of an INT8 tile
constexpr int FIRST_EPI = 4, EPI_WARPS = 8, FIRST_DEC = FIRST_EPI + EPI_WARPS, DEC_WARPS = 16;
constexpr int PITCH = 80;                          // staged row piece: 32 columns FP16 + pad

// A stage of the ring is a k-block of MT activation tiles and one weight tile, with a barrier each
// for "activations landed", "weights there" (copied, or decoded) and "multiplied".  Only its own
// copies complete a barrier that a copying warp waits for before it leaves: had the activations one
// with the decode warps, and had those given up, that wait would run to its limit for every stage.
template <int FMT, int MT>
struct Layout {
  static constexpr int THREADS = (FMT == 0 ? FIRST_DEC : FIRST_DEC + DEC_WARPS) * 32;
  static constexpr int CODE_ROW = FMT == 1 ? 64 : (FMT == 2 ? 32 : 0);
  static constexpr int CODES = BN * CODE_ROW;
  static constexpr int STAGE = (MT + 1) * TILE;                // activations, then weights
  static constexpr int S = FMT == 0 ? (MT == 2 ? 4 : 6) : (MT == 2 ? 3 : 4);
  static constexpr int SC = FMT == 0 ? 1 : (FMT == 1 ? 4 : 8); // packed codes
  static constexpr int BUFS = 2;                               // accumulator sets in TMEM
  static constexpr int COPIES = 16;
  // Groups of decode warps, which take k-blocks in turn.  A group waits for a stage by the parity
  // of its barrier, which tells one use from the next but not from the one after that.  With no
  // more groups than stages no group is two uses ahead: its own k-block c - GROUPS went into a
  // stage that c - GROUPS - S had left, and with that every k-block up to c - 2 S.  A slab of codes
  // is always the same group's.
  static constexpr int GROUPS = FMT == 2 && S >= 4 ? 4 : 2, GROUP_WARPS = DEC_WARPS / GROUPS;
  static_assert(FMT == 0 || (GROUPS <= S && SC % GROUPS == 0), "parities of the rings");
  static constexpr int TABLES = FMT == 0 ? 0 : static_cast<int>(sizeof(E8pLut<COPIES>));
  static constexpr int CODE_OFF = S * STAGE;
  static constexpr int TABLE_OFF = CODE_OFF + SC * CODES;
  static constexpr int OUT_OFF = TABLE_OFF + TABLES;           // epilogue: staged rows
  static constexpr int SCALE_OFF = OUT_OFF + EPI_WARPS * 16 * PITCH;   // 64 columns per warp
  static constexpr int BAR_OFF = SCALE_OFF + EPI_WARPS * 256;
  static constexpr int LIST_OFF = BAR_OFF + 512;
  static constexpr int LIST_ROOM = (226 * 1024 - LIST_OFF) / 8;
  static constexpr int TOTAL = 227 * 1024;                     // with 1 KB to align
  static_assert(LIST_ROOM >= 512, "exceeds the shared memory of one CTA");
};

struct Args {
  const unsigned char* w;
  const float* a_scale;
  const __half* w_scale;
  __half* out;
  int M, N, K, n_end;
  const int* tiles;             // expert tile table (see moe.cu), nullptr: an ordinary product
  const int* meta;
  long long w_stride;
};

struct Tile {
  int n0, m0, m_limit, expert, mt_act;
};

template <int FMT, int MT>
__global__ void __launch_bounds__(Layout<FMT, MT>::THREADS, 1) qgemm_walk_kernel(
    const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
    const __grid_constant__ Args p, const E8pTables* __restrict__ tables, int* status) {
  using L = Layout<FMT, MT>;
  constexpr int S = L::S, SC = L::SC, BUFS = L::BUFS;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* code_s = smem + L::CODE_OFF;
  using Lut = E8pLut<L::COPIES>;
  Lut* lut = reinterpret_cast<Lut*>(smem + L::TABLE_OFF);
  float* scale_s = reinterpret_cast<float*>(smem + L::SCALE_OFF);
  int2* list = reinterpret_cast<int2*>(smem + L::LIST_OFF);    // first row, expert and rows
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* a_full = bars;                     // [S]    activations of a stage landed
  uint64_t* full = a_full + S;                 // [S]    its weights landed or decoded
  uint64_t* empty = full + S;                  // [S]    its MMAs retired
  uint64_t* c_full = empty + S;                // [SC]   packed codes landed
  uint64_t* c_empty = c_full + SC;             // [SC]   every decode warp has read them
  uint64_t* acc_full = c_empty + SC;           // [BUFS] all MMAs of a tile retired
  uint64_t* acc_empty = acc_full + BUFS;       // [BUFS] accumulators read out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + BUFS);
  volatile int* abort_w = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* hits = reinterpret_cast<int*>(tmem_slot + 2);           // [32]
  static_assert((3 * S + 2 * SC + 2 * BUFS) * 8 + 8 + 128 <= 512, "barriers");

  const int tid = threadIdx.x, warp = warp_same(tid >> 5), lane = tid & 31;
  if (p.tiles != nullptr) grid_wait();          // the table
  const int n_tiles = (p.n_end + BN - 1) / BN, kblocks = p.K / BK;
  int m_tiles = (p.M + BM * MT - 1) / (BM * MT);
  if (p.tiles != nullptr) {
    // MT neighbouring 128-row tiles of one expert are one tile here (the fourth word counts an
    // expert's tiles)
    const int entries = p.meta[0];
    const int4* table = reinterpret_cast<const int4*>(p.tiles);
    int count = 0;
    for (int base = 0; base < entries; base += L::THREADS) {
      const int t = base + tid;
      int4 e = make_int4(0, 0, 0, 1);
      if (t < entries) e = table[t];
      const bool hit = t < entries && e.w % MT == 0;
      const unsigned ballot = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) hits[warp] = __popc(ballot);
      __syncthreads();
      int at = count + __popc(ballot & ((1u << lane) - 1u));
#pragma unroll 1
      for (int q = 0; q < L::THREADS / 32; ++q) {
        at += q < warp ? hits[q] : 0;
        count += hits[q];
      }
      if (hit && at < L::LIST_ROOM) {
        int rows = e.z;
#pragma unroll
        for (int i = 1; i < MT; ++i)
          if (t + i < entries && table[t + i].x == e.x) rows += table[t + i].z;
        list[at] = make_int2(e.y, e.x * 512 + rows);
      }
      __syncthreads();
    }
    m_tiles = min(count, L::LIST_ROOM);
  }
  const int total = warp_same(n_tiles * m_tiles);
  auto tile_at = [&](int t) {
    Tile T;
    const int nt = t / m_tiles, mi = t - nt * m_tiles;
    T.n0 = nt * BN;
    T.expert = 0;
    T.m0 = mi * BM * MT;
    T.m_limit = p.M;
    if (p.tiles != nullptr) {
      const int2 e = list[mi];
      T.expert = e.y >> 9;
      T.m0 = e.x;
      T.m_limit = e.x + (e.y & 511);
    }
    T.mt_act = min(MT, (T.m_limit - T.m0 + BM - 1) / BM);
    return T;
  };

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&full[s], FMT == 0 ? 1 : L::GROUP_WARPS);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < SC; ++s) {
      mbar_init(&c_full[s], 1);
      mbar_init(&c_empty[s], L::GROUP_WARPS);
    }
    for (int b = 0; b < BUFS; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], EPI_WARPS);
    }
    *abort_w = 0;
    mbar_fence_init();
    prefetch_tmap(&tmap_a);
    if (FMT == 0) prefetch_tmap(&tmap_b);
  }
  constexpr uint32_t TMEM_COLS = BUFS * MT * BN;
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  if (FMT != 0 && warp >= FIRST_DEC)
    e8p_lut_init(lut, tables, tid - FIRST_DEC * 32, DEC_WARPS * 32);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_same(*tmem_slot);
  grid_wait();
  grid_release();

#define WALK_WAIT(bar, par, code, detail) \
  mbar_wait_abortable((bar), (par), status, (code), (detail), abort_w)

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0, issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < total; t += gridDim.x) {
        const Tile T = tile_at(t);
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = WALK_WAIT(&empty[s], phase ^ 1, STATUS_TMA_WAIT, kb);
          if (!ok) break;
          mbar_expect_tx(&a_full[s], T.mt_act * TILE);
#pragma unroll
          for (int i = 0; i < MT; ++i)
            if (i < T.mt_act)
              tma_load_2d(smem + s * L::STAGE + i * TILE, &tmap_a, &a_full[s], kb * BK,
                          T.m0 + i * BM);
          ++issued;
          if (++s == S) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      // no copy of ours is in flight when the CTA ends
      for (uint32_t c = issued > S ? issued - S : 0; c < issued; ++c)
        mbar_wait(&a_full[c % S], (c / S) & 1, status, STATUS_TMA_WAIT, 0x4000);
    }
  } else if (warp == 2) {
    if (lane == 0) {
      constexpr int DEPTH = FMT == 0 ? S : SC;
      uint64_t* landed = FMT == 0 ? full : c_full;
      uint64_t* freed = FMT == 0 ? empty : c_empty;
      int s = 0;
      uint32_t phase = 0, issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < total; t += gridDim.x) {
        const Tile T = tile_at(t);
        const uint32_t bytes = min(BN, p.n_end - T.n0) * L::CODE_ROW;
        const unsigned char* src = p.w + T.expert * p.w_stride +
                                   static_cast<size_t>(T.n0) * L::CODE_ROW;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = WALK_WAIT(&freed[s], phase ^ 1, STATUS_TMA_WAIT, 0x1000 | kb);
          if (!ok) break;
          if (FMT == 0) {
            mbar_expect_tx(&full[s], TILE);
            tma_load_2d(smem + s * L::STAGE + MT * TILE, &tmap_b, &full[s], kb * BK,
                        T.expert * p.N + T.n0);
          } else {
            mbar_expect_tx(&c_full[s], bytes);
            bulk_load(code_s + s * L::CODES, src, bytes, &c_full[s]);
            src += static_cast<size_t>(p.N) * L::CODE_ROW;
          }
          ++issued;
          if (++s == DEPTH) {
            s = 0;
            phase ^= 1;
          }
        }
      }
      for (uint32_t c = issued > DEPTH ? issued - DEPTH : 0; c < issued; ++c)
        mbar_wait(&landed[c % DEPTH], (c / DEPTH) & 1, status, STATUS_TMA_WAIT, 0x5000);
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc(2, 1, 1, 0, 0, BM, BN);
    const uint32_t leader = elect_one();
    const uint64_t ring = umma_desc(smem_u32(smem), 16, 1024);
    int s = 0;
    uint32_t phase = 0, it = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < total; t += gridDim.x, ++it) {
      const int mt_act = warp_same(tile_at(t).mt_act);
      const uint32_t buf = it % BUFS, acc = tmem_base + buf * MT * BN;
      // the epilogue has read out what these accumulators held before
      if (it >= BUFS)
        ok = warp_all(
            WALK_WAIT(&acc_empty[buf], (it / BUFS - 1) & 1, STATUS_MMA_WAIT, 0x3000));
      for (int kb = 0; ok && kb < kblocks; ++kb) {
        ok = warp_all(WALK_WAIT(&full[s], phase, STATUS_MMA_WAIT, 0x2000 | kb) &&
                      WALK_WAIT(&a_full[s], phase, STATUS_MMA_WAIT, kb));
        if (!ok) break;
        tc_fence_after();
        const uint64_t ad = ring + static_cast<uint64_t>(s * L::STAGE / 16);
        const uint64_t bd = ad + MT * TILE / 16;
#pragma unroll
        for (int j = 0; j < BK / 32; ++j) {
#pragma unroll
          for (int i = 0; i < MT; ++i)
            if (i == 0 || i < mt_act)
              mma_i8_ss_by(leader, acc + i * BN, ad + (i * TILE + j * 32) / 16, bd + j * 32 / 16,
                           idesc, (kb | j) != 0 ? 1u : 0u);
        }
        tc_commit_by(leader, &empty[s]);
        if (++s == S) {
          s = 0;
          phase ^= 1;
        }
      }
      if (ok) tc_commit_by(leader, &acc_full[buf]);
    }
    __syncwarp();
  } else if (warp >= FIRST_EPI && warp < FIRST_DEC) {
    // ---------------- epilogue: a warp reads 32 rows x 64 columns of every accumulator
    const int quad = warp & 3, half = (warp - FIRST_EPI) >> 2;
    const int row = quad * 32 + lane;
    float* ws = scale_s + (warp - FIRST_EPI) * 64;
    unsigned char* stage = smem + L::OUT_OFF + (warp - FIRST_EPI) * 16 * PITCH;
    uint32_t it = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < total; t += gridDim.x, ++it) {
      const Tile T = tile_at(t);
      const uint32_t buf = it % BUFS;
      const int nw = T.n0 + half * 64;
      float sa[MT];
#pragma unroll
      for (int s = 0; s < MT; ++s) {
        const int m = T.m0 + s * BM + row;
        sa[s] = m < T.m_limit ? p.a_scale[m] : 0.f;
      }
      float2 w2 = make_float2(0.f, 0.f);
      if (nw + lane * 2 < p.n_end)
        w2 = __half22float2(*reinterpret_cast<const __half2*>(
            p.w_scale + static_cast<size_t>(T.expert) * p.N + nw + lane * 2));
      __syncwarp();
      reinterpret_cast<float2*>(ws)[lane] = w2;
      ok = WALK_WAIT(&acc_full[buf], (it / BUFS) & 1, STATUS_EPILOGUE_WAIT, 0);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < MT; ++s) {
        const bool used = s < T.mt_act;
        const uint32_t acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                             (buf * MT + s) * BN + half * 64;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t r[32];
          if (used) {
            tmem_ld_32x32(acc + c * 32, r);
            tc_wait_ld();
          }
          if (s == MT - 1 && c == 1) {             // this warp's share is in registers
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
          }
          if (!used) continue;
          uint32_t h[16];                          // the row's 32 columns
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 x = *reinterpret_cast<const float4*>(ws + c * 32 + g * 4);
            const __half2 lo = __floats2half2_rn(
                (static_cast<float>(static_cast<int>(r[g * 4])) * x.x) * sa[s],
                (static_cast<float>(static_cast<int>(r[g * 4 + 1])) * x.y) * sa[s]);
            const __half2 hi = __floats2half2_rn(
                (static_cast<float>(static_cast<int>(r[g * 4 + 2])) * x.z) * sa[s],
                (static_cast<float>(static_cast<int>(r[g * 4 + 3])) * x.w) * sa[s]);
            h[g * 2] = *reinterpret_cast<const uint32_t*>(&lo);
            h[g * 2 + 1] = *reinterpret_cast<const uint32_t*>(&hi);
          }
          const int seg = lane & 3, n = nw + c * 32 + seg * 8;
          __half* dst = p.out + static_cast<size_t>(T.m0 + s * BM + quad * 32) * p.N + n;
          const int rows = T.m_limit - (T.m0 + s * BM + quad * 32);
#pragma unroll
          for (int b = 0; b < 2; ++b) {            // sixteen rows at a time through the stage
            __syncwarp();
            if (lane >> 4 == b) {
#pragma unroll
              for (int g = 0; g < 4; ++g)
                *reinterpret_cast<uint4*>(stage + (lane & 15) * PITCH + g * 16) =
                    make_uint4(h[g * 4], h[g * 4 + 1], h[g * 4 + 2], h[g * 4 + 3]);
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int rr = i * 8 + (lane >> 2);
              if (b * 16 + rr < rows && n + 8 <= p.n_end)
                *reinterpret_cast<int4*>(dst + static_cast<size_t>(b * 16 + rr) * p.N) =
                    *reinterpret_cast<const int4*>(stage + rr * PITCH + seg * 16);
            }
          }
        }
      }
    }
  } else if (FMT != 0 && warp >= FIRST_DEC) {
    // ---------------- lattice decode: a group's rows of 16 bytes x 8 threads per pass
    constexpr int STEP = L::GROUP_WARPS * 4, PASSES = BN / STEP;
    const int t = tid - FIRST_DEC * 32, chunk = t & 7, first = (t >> 3) % STEP;
    const E8pLane<L::COPIES> look(lut, lane);
    const int me = blockIdx.x, ctas = gridDim.x;
    const int own_tiles = total > me ? (total - 1 - me) / ctas + 1 : 0;
    const uint32_t all = static_cast<uint32_t>(own_tiles) * kblocks;
    for (uint32_t cb = (warp - FIRST_DEC) / L::GROUP_WARPS; cb < all; cb += L::GROUPS) {
      const uint32_t sc = cb % SC, sb = cb % S;
      bool ok = warp_all(WALK_WAIT(&c_full[sc], (cb / SC) & 1, STATUS_DECODE_WAIT, cb & 0x7ff));
      if (!ok) break;
      const unsigned char* cs = code_s + sc * L::CODES;
      uint2 word[PASSES];
      uint32_t seen = 0;
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int row = first + STEP * i;
        word[i] = make_uint2(0u, 0u);
        if (FMT == 1) word[i] = *reinterpret_cast<const uint2*>(cs + row * 64 + chunk * 8);
        else word[i].x = *reinterpret_cast<const uint32_t*>(cs + row * 32 + chunk * 4);
        seen ^= word[i].x ^ word[i].y;
      }
      ok = warp_all(WALK_WAIT(&empty[sb], ((cb / S) & 1) ^ 1, STATUS_DECODE_WAIT,
                              0x800 | (cb & 0x7ff)));
      if (!ok) break;
      unsigned char* bs = smem + sb * L::STAGE + MT * TILE;
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int row = first + STEP * i;
        uint2 x, y;
        if constexpr (FMT == 1) {
          x = e8p_decode_q4(word[i].x, look);
          y = e8p_decode_q4(word[i].y, look);
        } else {
          x = e8p_decode_q2<0>(word[i].x, look);
          y = e8p_decode_q2<1>(word[i].x, look);
        }
        // (rows past the matrix: their codes are stale, their products are not stored)
        *reinterpret_cast<uint4*>(bs + swz128(row, chunk)) = make_uint4(x.x, x.y, y.x, y.y);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[sb]);
      hand_back(&c_empty[sc], seen);
    }
  }
#undef WALK_WAIT
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

template <int FMT, int MT>
int launch(const WalkCall& c, cudaStream_t stream) {
  using L = Layout<FMT, MT>;
  if (c.tiles != nullptr && c.max_tiles > L::LIST_ROOM) return -1;
  CUtensorMap ta, tb;
  if (!make_tmap_2d(&ta, c.a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, c.M, c.K, c.K, BM, BK)) return -3;
  if (FMT == 0) {
    if (!make_tmap_2d(&tb, c.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1,
                      static_cast<uint64_t>(c.N) * c.experts, c.K, c.K, BN, BK))
      return -3;
  } else {
    tb = ta;
    if (reinterpret_cast<uintptr_t>(c.w) % 16) return -1;
  }
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, qgemm_walk_kernel<FMT, MT>, L::TOTAL)) return e;
  const long tiles = static_cast<long>((c.n_end + BN - 1) / BN) *
                     (c.tiles ? c.max_tiles : (c.M + BM * MT - 1) / (BM * MT));
  const Args p{static_cast<const unsigned char*>(c.w), c.a_scale, c.w_scale, c.out, c.M, c.N, c.K,
               c.n_end, c.tiles, c.meta, c.w_stride};
  launch_early(qgemm_walk_kernel<FMT, MT>, static_cast<unsigned>(tiles < 148 ? tiles : 148),
               L::THREADS, L::TOTAL, stream, ta, tb, p, runtime_e8p_tables(), runtime_status_ptr());
  return static_cast<int>(cudaGetLastError());
}

}  // namespace walk

int walk_list_room(int fmt) {
  return fmt == 0   ? walk::Layout<0, 2>::LIST_ROOM
         : fmt == 1 ? walk::Layout<1, 2>::LIST_ROOM
                    : walk::Layout<2, 2>::LIST_ROOM;
}

int qgemm_walk_dispatch(int fmt, int mt, const WalkCall& c, cudaStream_t stream) {
  if (fmt == 0) return mt == 2 ? walk::launch<0, 2>(c, stream) : walk::launch<0, 1>(c, stream);
  if (fmt == 1) return mt == 2 ? walk::launch<1, 2>(c, stream) : walk::launch<1, 1>(c, stream);
  return mt == 2 ? walk::launch<2, 2>(c, stream) : walk::launch<2, 1>(c, stream);
}

}  // namespace orinfer
