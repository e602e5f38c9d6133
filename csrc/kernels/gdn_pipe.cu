// Gated delta rule over long runs, one CTA of sixteen warps per SM: the chunked form of gdn.cu
// (the same sums: see gdn_chunk_kernel for the mathematics and how each product keeps FP32
// accuracy) as a pipeline of roles.  In a round
//   * eight state warps take one chunk.  A warp owns eight value channels: S (128 x 8) stays in
//     its accumulators, and as the B operand of the next chunk's products it goes through shared
//     memory, split into FP16 halves as it is made;
//   * four output warps form the outputs of the chunk before, from that copy of S and from Delta;
//   * one warp each makes P of this chunk, T of the next, A of the one after and the gates ahead
//     of that.
// gdn_chunk_kernel, whose four warps carry the state and form the outputs, waits for its chain of
// some 2000 instructions a chunk and fills 30 % of the issue slots; two of its CTAs fit an SM and
// hide each other.  Here the chain is a third as long.  What bounds a round (about 6300 cycles) is
// shared memory (its pipe is busy for 4300 of them: operands, the k rows once per eight channels)
// and the state warps' chain; issue slots are 45 % in use, the tensor core 37 %.  On the way: code
// that does not stay in the instruction cache cost most (T, P and A unrolled: 8500 cycles a round,
// rolled 6300); all loads ahead, four sums in turn instead of two, state and output warps on
// schedulers of their own, or outputs held back until S^T k is through: no change.  32 heads of 128
// channels, with the convolution and the norm of then: one run of 1050 rows 205 -> 155 us, two 245
// -> 181, one of 4000 725 -> 547, two of 250 71 -> 54, two of 64 29.1 -> 24.5, one of 40 24.4 ->
// 21.
// With more CTAs than SMs, two waves of these stand against one of two per SM: three runs of 40
// rows 31 against 37, of 250 88 against 94, sixteen of 64 115 against 127, and from some 400 rows
// on these win again (three of 1000 337 -> 315, eight of 500 364 -> 349).
#include "api.h"
#include "common.cuh"
#include "gdn_chunk.cuh"

namespace orinfer {
namespace pipe {

// As mma16816 and mma_tf32, but free to be moved among other products: a sum waits 22 cycles for
// the product before, and others fit between.
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                        uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_t32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                        uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int STATE_WARPS = 8, OUT_WARPS = 4;
constexpr int THREADS = (STATE_WARPS + OUT_WARPS + 4) * 32;
constexpr int FRAG = 144;                      // floats of a stored 16 x 8 operand tile (padded)
struct Smem {
  __half k[4][CHUNK][136], q[3][CHUNK][136];   // rows padded to 17 16-byte units (ldmatrix)
  __half v[2][CHUNK][72];
  __half s[2][STATE_WARPS][2][128][8];         // S before a chunk: head and remainder, [dk][dv]
  float down[2][STATE_WARPS][8];               // and the power of two of each value channel
  float d[2][STATE_WARPS][CHUNK][12];          // B, then Delta: [row][dv], rows padded
  float t[2][2][8][FRAG], p[2][2][8][FRAG];    // T and P below the diagonal, TF32 pairs
  float at[2][CHUNK][36];                      // A transposed: [j][i]
  float tx[CHUNK][32];                         // T as it is made, a column per lane
  float pd[2][CHUNK];                          // diagonal of P (that of T is 1)
  float gh[8][CHUNK], gl[8][CHUNK], eg[8][CHUNK], beta[8][CHUNK], tail[8][CHUNK], total[8];
  float k_max[8];                              // largest magnitude among a chunk's k
};
// Where element (i, j) of a 32 x 32 matrix lies among the stored operand tiles: tile (i / 16, j /
// 8) in the order of an m16n8k8 A operand whose k index t is column 2t and whose t + 4 is 2t + 1,
// so that a lane's four words are one 16-byte load.
__device__ __forceinline__ int frag_at(int i, int j) {
  return ((i >> 4) * 4 + (j >> 3)) * FRAG + (i & 7) * 16 + ((j & 7) >> 1) * 4 + ((i >> 3) & 1) +
         2 * (j & 1);
}

// FP16 head and remainder of two values (already scaled into the FP16 range)
__device__ __forceinline__ float2 split_head(float2 x, uint32_t& hi) {     // what the head leaves
  const __half2 h = __floats2half2_rn(x.x, x.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  return fma2(__half22float2(h), make_float2(-1.f, -1.f), x);
}
__device__ __forceinline__ void split_half2(float2 x, uint32_t& hi, uint32_t& lo) {
  const float2 rest = split_head(x, hi);
  const __half2 l = __floats2half2_rn(rest.x, rest.y);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split_half3(float2 x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  split_half2(split_head(x, hi), mid, lo);
}
// The same with the remainder 2^11 times as large, so that its smallest step is 2^-35, not 2^-24
constexpr float REST_UP = 2048.f;
__device__ __forceinline__ void split_state(float2 x, uint32_t& hi, uint32_t& lo) {
  const float2 rest = mul2(split_head(x, hi), make_float2(REST_UP, REST_UP));
  const __half2 l = __floats2half2_rn(rest.x, rest.y);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// d += a, two by two
__device__ __forceinline__ void add4(float (&d)[4], const float (&a)[4]) {
  const float2 x = add2(make_float2(d[0], d[1]), make_float2(a[0], a[1]));
  const float2 y = add2(make_float2(d[2], d[3]), make_float2(a[2], a[3]));
  d[0] = x.x; d[1] = x.y; d[2] = y.x; d[3] = y.y;
}

// D (32 x 8, two 16-row MMA tiles) += M X for N such D and X: M a 32 x 32 matrix below the
// diagonal, stored as TF32 pairs (m[0] heads, m[1] remainders), X [row][channel] in shared memory,
// split here. A zero does not hide an infinity or a NaN of a later row in a tensor-core product,
// so where the warp's X hold one (`wild`) the sums are made term by term and earlier rows stay as
// they are.
template <int N>
__device__ __forceinline__ void mul_lower(float (&d)[N][2][4], const float (*m)[8][FRAG],
                                          const float (*x)[CHUNK][12], bool wild, int lane) {
  const int g = lane >> 2, t = lane & 3;
  if (wild) {
    const float *head = &m[0][0][0], *rest = &m[1][0][0];
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 16 * (e >> 2) + 8 * ((e >> 1) & 1) + g, col = 2 * t + (e & 1);
        float sum = d[n][e >> 2][e & 3];
#pragma unroll 1
        for (int j = 0; j < i; ++j)
          sum = fmaf(head[frag_at(i, j)] + rest[frag_at(i, j)], x[n][j][col], sum);
        d[n][e >> 2][e & 3] = sum;
      }
    return;
  }
  uint32_t xh[N][4][2], xl[N][4][2];
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int e = 0; e < 2; ++e) split_tf32(x[n][8 * s + 2 * t + e][g], xh[n][s][e], xl[n][s][e]);
  // tiles (i, s) in two groups of three, whose products take turns: a product waits 22 cycles for
  // the one before it in the same sum
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t hi[3][4], lo[3][4];
    float part[N][3][4] = {};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int tile = q == 0 ? (k == 0 ? 0 : k == 1 ? 1 : 4) : 5 + k;
      const uint4 h4 = *reinterpret_cast<const uint4*>(&m[0][tile][lane * 4]);
      const uint4 l4 = *reinterpret_cast<const uint4*>(&m[1][tile][lane * 4]);
      hi[k][0] = h4.x; hi[k][1] = h4.y; hi[k][2] = h4.z; hi[k][3] = h4.w;
      lo[k][0] = l4.x; lo[k][1] = l4.y; lo[k][2] = l4.z; lo[k][3] = l4.w;
    }
#pragma unroll
    for (int step = 0; step < 3; ++step)
#pragma unroll
      for (int n = 0; n < N; ++n)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int s = q == 0 ? k & 1 : 1 + k;
          mma_t32(part[n][k], step == 1 ? lo[k] : hi[k], step == 0 ? xl[n][s][0] : xh[n][s][0],
                   step == 0 ? xl[n][s][1] : xh[n][s][1]);
        }
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int k = 0; k < 3; ++k) add4(d[n][q == 0 && k < 2 ? 0 : 1], part[n][k]);
  }
}

// D (32 x 8) = X S for N such D and slices of S: X a chunk's rows of k or q, S as `s` holds it. The
// remainders' sums are scaled back before those of the heads (under 1 % of a run; sums of their own
// took 4 %, heads and remainders made behind the true maximum 2 %).
template <int N, int UNROLL>
__device__ __forceinline__ void mul_state(float (&d)[N][2][4], const __half (*x)[136],
                                          const __half (*s)[2][128][8], int lane) {
  const int mat = lane >> 3, mrow = lane & 7;
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) d[n][m][e] = 0.f;
#pragma unroll UNROLL
  for (int u = 0; u < 4; ++u) {                    // 32 key channels
    uint32_t f[N][2][4], a[2][2][4];               // remainders and heads; [row tile][half]
#pragma unroll
    for (int n = 0; n < N; ++n) ldsm_x4_t(f[n][0], &s[n][1][32 * u + lane][0]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const __half* at = &x[16 * m + (mat & 1) * 8 + mrow][32 * u + (mat >> 1) * 8];
      ldsm_x4(a[m][0], at);
      ldsm_x4(a[m][1], at + 16);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) ldsm_x4_t(f[n][1], &s[n][0][32 * u + lane][0]);
    float part[N][2][4] = {};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int m = 0; m < 2; ++m)              // the sums take turns
            mma_f16(part[n][m], a[m][k][0], a[m][k][1], a[m][k][2], a[m][k][3], f[n][w][2 * k],
                    f[n][w][2 * k + 1]);
      if (w == 0) {
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int e = 0; e < 8; ++e) part[n][e >> 2][e & 3] *= 1.f / REST_UP;
      }
    }
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int m = 0; m < 2; ++m) add4(d[n][m], part[n][m]);
  }
}

// Sixteen rows, 16 i on, of X K^T (X rows of k or q) times e^(G_i - G_j), as far as the diagonal:
// two or four 16 x 8 tiles.  G comes as FP32 pairs: differences of the heads round in proportion
// to themselves, and the remainders restore what the heads lost.
__device__ __forceinline__ void mul_keys(float (&acc)[4][4], const __half (*x)[136],
                                         const __half (*k)[136], const float* gh, const float* gl,
                                         int i, int lane) {
  const int g = lane >> 2, t = lane & 3, tiles = 2 * i + 2;
  const __half* xa = &x[16 * i + (lane >> 3 & 1) * 8 + (lane & 7)][(lane >> 4) * 8];
  const __half* kb = &k[lane & 7][(lane >> 3) * 8];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {                      // sums of 16 channels, two at a time
    uint32_t a[2][4];
    float d[2][4][4] = {};
    ldsm_x4(a[0], xa + 32 * s);
    ldsm_x4(a[1], xa + 32 * s + 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j >= tiles) break;
      uint32_t b[4];
      ldsm_x4(b, kb + j * 8 * 136 + 32 * s);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        mma_f16(d[h][j], a[h][0], a[h][1], a[h][2], a[h][3], b[2 * h], b[2 * h + 1]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      add4(acc[j], d[0][j]);
      add4(acc[j], d[1][j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (j >= tiles) break;
    const float2 ch = *reinterpret_cast<const float2*>(&gh[8 * j + 2 * t]);
    const float2 cl = *reinterpret_cast<const float2*>(&gl[8 * j + 2 * t]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float rh = gh[16 * i + 8 * h + g], rl = gl[16 * i + 8 * h + g];
      acc[j][2 * h] *= expf(fminf((rh - ch.x) + (rl - cl.x), 0.f));
      acc[j][2 * h + 1] *= expf(fminf((rh - ch.y) + (rl - cl.y), 0.f));
    }
  }
}

// all warps of the CTA, each from its own loop
__device__ __forceinline__ void round_end() { asm volatile("bar.sync 0;" ::: "memory"); }

__global__ void __launch_bounds__(THREADS, 1) gdn_pipe_kernel(
    const __half* __restrict__ qkv, int conv_dim, const float* __restrict__ ab,
    const float* __restrict__ a_log, const float* __restrict__ dt_bias,
    const Segment* __restrict__ segs, const int* __restrict__ row_slot,
    const int* __restrict__ row_pos, int hk, int hv, float* __restrict__ state,
    float* __restrict__ out) {
  constexpr int D = 128;
  extern __shared__ __align__(16) unsigned char pipe_smem[];
  Smem& sm = *reinterpret_cast<Smem*>(pipe_smem);
  grid_release();
  const Segment seg = segs[blockIdx.y];
  if (seg.rows < GDN_LONG_ROWS) return;
  const int vh = blockIdx.x >> 1, kh = vh / (hv / hk), dk_total = hk * D;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int mat = lane >> 3, mrow = lane & 7;          // this lane's row in an ldmatrix
  const int dv0 = (blockIdx.x & 1) * 64;
  const int chunks = (seg.rows + CHUNK - 1) / CHUNK;
  const float scale = rsqrtf(static_cast<float>(D));

  // In round r the state warps take chunk r, the output warps chunk r - 1, and ahead of them P is
  // made of chunk r, T of chunk r + 1, A of chunk r + 2 and the gates of chunk r + 3, while k of
  // that chunk and q and v of chunk r + 1 are copied in.
  if (warp < STATE_WARPS) {
    // ---- S, rows dk = 16 i + g (+ 8), value channels 2t and 2t + 1 of this warp's eight
    const bool fresh = row_pos[seg.row_start] == 0;
    float* sp = state + (static_cast<size_t>(row_slot[seg.row_start]) * hv + vh) * D * D + dv0 +
                warp * 8 + 2 * t;
    float s_acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float2 x = make_float2(0.f, 0.f);
        if (!fresh) x = *reinterpret_cast<const float2*>(sp + (16 * i + 8 * h + g) * D);
        s_acc[i][2 * h] = x.x;
        s_acc[i][2 * h + 1] = x.y;
      }
    float s_max[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) s_max[e & 1] = fmaxf(s_max[e & 1], fabsf(s_acc[i][e]));
    // S as the products read it: FP16 halves under a power of two per value channel, `e` above all
    float2 up, down;
    auto scale_to = [&](const float (&bound)[2], int next) {
      const int e0 = bound_exp(bound[0]), e1 = bound_exp(bound[1]);
      up = make_float2(pow2i(14 - e0), pow2i(14 - e1));
      down = make_float2(pow2i(e0 - 14), pow2i(e1 - 14));
      if (g == 0) *reinterpret_cast<float2*>(&sm.down[next][warp][2 * t]) = down;
    };
    auto place = [&](int i, int next) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t hi, lo;
        split_state(mul2(make_float2(s_acc[i][2 * h], s_acc[i][2 * h + 1]), up), hi, lo);
        *reinterpret_cast<uint32_t*>(&sm.s[next][warp][0][16 * i + 8 * h + g][2 * t]) = hi;
        *reinterpret_cast<uint32_t*>(&sm.s[next][warp][1][16 * i + 8 * h + g][2 * t]) = lo;
      }
    };
    auto all_rows = [&] {                              // the maxima over the lanes of a column
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int o = 4; o < 32; o <<= 1)
          s_max[h] = fmaxf(s_max[h], __shfl_xor_sync(0xffffffffu, s_max[h], o));
    };
    all_rows();
    scale_to(s_max, 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) place(i, 0);
    for (int r = -3; r < 0; ++r) round_end();
    for (int c = 0; c < chunks; ++c) {
      const int buf = c & 1, ring = c & 7;
      __syncwarp();
      // ---- S^T k, then B
      float x1[1][2][4];
      float(&x)[2][4] = x1[0];
      mul_state<1, 2>(x1, sm.k[c & 3], &sm.s[buf][warp], lane);
      float(*xs)[12] = sm.d[buf][warp];
      float size = 0.f;
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = 16 * m + 8 * h + g;
          const float eg = sm.eg[ring][row], be = sm.beta[ring][row];
          const float2 v = __half22float2(
              *reinterpret_cast<const __half2*>(&sm.v[buf][row][warp * 8 + 2 * t]));
          float2 b;
          b.x = be * fmaf(-(eg * down.x), x[m][2 * h], v.x);
          b.y = be * fmaf(-(eg * down.y), x[m][2 * h + 1], v.y);
          x[m][2 * h] = b.x;
          x[m][2 * h + 1] = b.y;
          *reinterpret_cast<float2*>(&xs[row][2 * t]) = b;
          size += fabsf(b.x) + fabsf(b.y);
        }
      const bool wild = __any_sync(0xffffffffu, !(size < INFINITY));
      __syncwarp();
      // ---- Delta: the diagonals carry most of both sums and are multiplied in FP32
      mul_lower<1>(x1, sm.t[buf], &sm.d[buf][warp], wild, lane);
      __syncwarp();
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(&xs[16 * m + 8 * h + g][2 * t]) =
              make_float2(x[m][2 * h], x[m][2 * h + 1]);
      __syncwarp();
      // ---- state update: rows 16 r + 8 h + 2t and the next, value channel g
      float dl[2][2][2], d_max = 0.f, d_sum = 0.f;
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = 16 * r + 8 * h + 2 * t;
          const float2 tl = *reinterpret_cast<const float2*>(&sm.tail[ring][row]);
          dl[r][h][0] = xs[row][g] * tl.x;
          dl[r][h][1] = xs[row + 1][g] * tl.y;
          d_max = fmaxf(d_max, fmaxf(fabsf(dl[r][h][0]), fabsf(dl[r][h][1])));
          d_sum += fabsf(dl[r][h][0]) + fabsf(dl[r][h][1]);
        }
      const int e = bound_exp(quad_max(d_max));
      const float dup = pow2i(14 - e), own_down = pow2i(e - 14);
      const float2 ddown2 = make_float2(__shfl_sync(0xffffffffu, own_down, 8 * t),
                                        __shfl_sync(0xffffffffu, own_down, 8 * t + 4));
      // head, remainder and its remainder: a new row of S is this product to the last bit
      uint32_t hi[2][2], mid[2][2], lo[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          split_half3(make_float2(dl[r][h][0] * dup, dl[r][h][1] * dup), hi[r][h], mid[r][h],
                      lo[r][h]);
      const float2 total2 = make_float2(sm.total[ring], sm.total[ring]);
      // The next S is split as it is made, under a bound of it: e^G S and the sum of the |Delta|
      // times the largest |k|, which can be half a dozen bits above its largest element.  Heads and
      // remainders have 2^49 steps below the bound, so an element keeps 22 bits down to 2^-27 of it
      // (gdn_chunk_kernel, whose remainders are not scaled up, down to 2^-16 of the largest).
      d_sum += __shfl_xor_sync(0xffffffffu, d_sum, 1);
      d_sum += __shfl_xor_sync(0xffffffffu, d_sum, 2);
      all_rows();
      const float k_max = 1.001f * sm.k_max[ring];
      const float bound[2] = {
          fmaf(__shfl_sync(0xffffffffu, d_sum, 8 * t), k_max, total2.x * s_max[0]),
          fmaf(__shfl_sync(0xffffffffu, d_sum, 8 * t + 4), k_max, total2.x * s_max[1])};
      // the output warps have read the S that this one replaces
      asm volatile("bar.sync 1, %0;" ::"n"((STATE_WARPS + OUT_WARPS) * 32) : "memory");
      scale_to(bound, buf ^ 1);
      s_max[0] = s_max[1] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        float add[2][2][4] = {};
        uint32_t a[2][2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            ldsm_x4_t(a[n][r],
                      &sm.k[c & 3][16 * r + (mat >> 1) * 8 + mrow][16 * (i + n) + (mat & 1) * 8]);
#pragma unroll
        for (int part = 0; part < 3; ++part)
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const uint32_t(&b)[2] = part == 0 ? lo[r] : part == 1 ? mid[r] : hi[r];
              mma_f16(add[n][r], a[n][r][0], a[n][r][1], a[n][r][2], a[n][r][3], b[0], b[1]);
            }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float(&y)[4] = s_acc[i + n];
            const float2 a0 = make_float2(add[n][0][2 * h], add[n][0][2 * h + 1]);
            const float2 a1 = make_float2(add[n][1][2 * h], add[n][1][2 * h + 1]);
            float2 v = fma2(make_float2(y[2 * h], y[2 * h + 1]), total2, mul2(a0, ddown2));
            v = fma2(a1, ddown2, v);
            y[2 * h] = v.x;
            y[2 * h + 1] = v.y;
            s_max[0] = fmaxf(s_max[0], fabsf(v.x));
            s_max[1] = fmaxf(s_max[1], fabsf(v.y));
          }
#pragma unroll
        for (int n = 0; n < 2; ++n) place(i + n, buf ^ 1);
      }
      round_end();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(sp + (16 * i + 8 * h + g) * D) =
            make_float2(s_acc[i][2 * h], s_acc[i][2 * h + 1]);
    round_end();
  } else if (warp < STATE_WARPS + OUT_WARPS) {
    // ---- outputs of two slices of eight channels a warp, and the copies: four threads a row; rows
    // past the run become zeros
    constexpr int N = STATE_WARPS / OUT_WARPS;
    const int w = warp - STATE_WARPS, copy_row = w * 8 + (lane >> 2), unit = (lane & 3) * 8;
    auto source = [&](int c) {
      const int n = min(CHUNK, seg.rows - c * CHUNK);
      const int row = seg.row_start + c * CHUNK + min(copy_row, n - 1);
      return qkv + static_cast<size_t>(row) * conv_dim + unit;
    };
    auto copy = [&](int c, __half* dst, const __half* src, int units) {
      const int bytes = c * CHUNK + copy_row < seg.rows ? 16 : 0;
#pragma unroll
      for (int i = 0; i < units; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + 32 * i)),
                     "l"(src + 32 * i), "r"(bytes)
                     : "memory");
    };
    auto state_read = [] {                             // S of the last chunk may be written over
      asm volatile("bar.arrive 1, %0;" ::"n"((STATE_WARPS + OUT_WARPS) * 32) : "memory");
    };
    for (int r = -3; r <= chunks; ++r) {
      if (r + 3 < chunks) {
        const int c = r + 3;
        copy(c, &sm.k[c & 3][copy_row][unit], source(c) + dk_total + kh * D, 4);
      }
      if (r >= -1 && r + 1 < chunks) {
        const int c = r + 1;
        copy(c, &sm.q[c % 3][copy_row][unit], source(c) + kh * D, 4);
        copy(c, &sm.v[c & 1][copy_row][unit], source(c) + 2 * dk_total + vh * D + dv0, 2);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (r == 0) state_read();
      if (r > 0) {
        const int c = r - 1, buf = c & 1, ring = c & 7;
        float x[N][2][4], size = 0.f;
        mul_state<N, 1>(x, sm.q[c % 3], &sm.s[buf][N * w], lane);
        float2 downs[N];
#pragma unroll
        for (int n = 0; n < N; ++n)
          downs[n] = *reinterpret_cast<const float2*>(&sm.down[buf][N * w + n][2 * t]);
        if (r < chunks) state_read();
#pragma unroll
        for (int n = 0; n < N; ++n) {
          const float2 down = downs[n];
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int row = 16 * m + 8 * h + g;
              const float2 dl = *reinterpret_cast<const float2*>(&sm.d[buf][N * w + n][row][2 * t]);
              const float eg = sm.eg[ring][row], pd = sm.pd[buf][row];
              float* y = &x[n][m][2 * h];
              y[0] = fmaf(pd, dl.x, y[0] * (eg * down.x * scale));
              y[1] = fmaf(pd, dl.y, y[1] * (eg * down.y * scale));
              size += fabsf(dl.x) + fabsf(dl.y);
            }
        }
        mul_lower<N>(x, sm.p[buf], &sm.d[buf][N * w], __any_sync(0xffffffffu, !(size < INFINITY)),
                     lane);
        const int rows = min(CHUNK, seg.rows - c * CHUNK);
        float* to = out + (static_cast<size_t>(seg.row_start + c * CHUNK) * hv + vh) * D + dv0 +
                    N * w * 8 + 2 * t;
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int row = 16 * m + 8 * h + g;
              if (row < rows)
                *reinterpret_cast<float2*>(to + static_cast<size_t>(row) * hv * D + 8 * n) =
                    make_float2(x[n][m][2 * h], x[n][m][2 * h + 1]);
            }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      round_end();
    }
  } else if (warp == STATE_WARPS + OUT_WARPS) {
    // ---- gates, three chunks ahead
    const float alog = expf(a_log[vh]), bias = dt_bias[vh];
    float n_a = 0.f, n_b = 0.f;
    auto fetch_gates = [&](int c) {
      const int r = c * CHUNK + lane;
      if (r < seg.rows) {
        const size_t row = static_cast<size_t>(seg.row_start + r);
        n_a = ab[row * 2 * hv + vh];
        n_b = ab[row * 2 * hv + hv + vh];
      }
    };
    fetch_gates(0);
    for (int r = -3; r <= chunks; ++r) {
      const int c = r + 3;
      if (c < chunks) {
        const int ring = c & 7;
        const bool live = c * CHUNK + lane < seg.rows;
        const float xg = n_a + bias;
        const float softplus = xg > 20.f ? xg : log1pf(expf(xg));
        // a decay that is zero in FP32 ends what a value was, also as the exponential of an
        // infinity: kept finite, so that differences of the sums stay defined (a NaN stays one)
        float log_decay = -alog * softplus;
        if (log_decay < -200.f) log_decay = -200.f;
        double big_g = live ? static_cast<double>(log_decay) : 0.0;
        const float beta = live ? __frcp_rn(1.f + expf(-n_b)) : 0.f;
        if (c + 1 < chunks) fetch_gates(c + 1);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double up = __shfl_up_sync(0xffffffffu, big_g, o);
          if (lane >= o) big_g += up;
        }
        const double last = __shfl_sync(0xffffffffu, big_g, 31);
        const float g_hi = static_cast<float>(big_g);
        sm.gh[ring][lane] = g_hi;
        sm.gl[ring][lane] = static_cast<float>(big_g - static_cast<double>(g_hi));
        sm.eg[ring][lane] = exp_pair(big_g);
        sm.beta[ring][lane] = beta;
        sm.tail[ring][lane] = exp_pair(last - big_g);
        if (lane == 0) sm.total[ring] = exp_pair(last);
      }
      if (r >= -2 && r + 2 < chunks) {                 // of the k that are there
        __half2 big = __half2half2(__ushort_as_half(0));
#pragma unroll 4
        for (int i = lane; i < CHUNK * 16; i += 32) {
          const uint4 u = *reinterpret_cast<const uint4*>(&sm.k[(r + 2) & 3][i >> 4][(i & 15) * 8]);
          const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
          for (int j = 0; j < 4; ++j) big = __hmax2(big, __habs2(h[j]));
        }
        const float2 both = __half22float2(big);
        const float all = warp_max(fmaxf(both.x, both.y));
        if (lane == 0) sm.k_max[(r + 2) & 7] = all;
      }
      round_end();
    }
  } else if (warp == STATE_WARPS + OUT_WARPS + 1) {
    // ---- A, two chunks ahead
    for (int r = -3; r <= chunks; ++r) {
      const int c = r + 2;
      if (c >= 0 && c < chunks) {
        const int ring = c & 7;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          float acc[4][4];
          mul_keys(acc, sm.k[c & 3], sm.k[c & 3], sm.gh[ring], sm.gl[ring], i, lane);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j >= 2 * i + 2) break;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int ri = 16 * i + (e >> 1) * 8 + g, cj = 8 * j + 2 * t + (e & 1);
              sm.at[c & 1][cj][ri] = cj < ri ? acc[j][e] * sm.beta[ring][ri] : 0.f;
            }
          }
        }
      }
      round_end();
    }
  } else if (warp == STATE_WARPS + OUT_WARPS + 2) {
    // ---- T: column `lane` by forward substitution, subtracting A's column j times T's row j,
    // eight rows at a time; the rows above them lie in shared memory, a lane's own column
    for (int r = -3; r <= chunks; ++r) {
      const int c = r + 1;
      if (c >= 0 && c < chunks) {
        const float(*at)[36] = sm.at[c & 1];
        float *head = &sm.t[c & 1][0][0][0], *rest = &sm.t[c & 1][1][0][0];
#pragma unroll 1
        for (int b = 0; b < CHUNK; b += 8) {
          float x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = b + i == lane ? 1.f : 0.f;
          auto subtract = [&](int j, float xj, int from) {
            const float4 a0 = *reinterpret_cast<const float4*>(&at[j][b]);
            const float4 a1 = *reinterpret_cast<const float4*>(&at[j][b + 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i >= from) x[i] = fmaf(-a[i], xj, x[i]);
          };
#pragma unroll 1
          for (int j = 0; j < b; j += 8)
#pragma unroll
            for (int u = 0; u < 8; ++u) subtract(j + u, sm.tx[j + u][lane], 0);
#pragma unroll
          for (int u = 0; u < 7; ++u) subtract(b + u, x[u], u + 1);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            sm.tx[b + i][lane] = x[i];
            uint32_t hi, lo;
            split_tf32(b + i == lane ? 0.f : x[i], hi, lo);
            head[frag_at(b + i, lane)] = __uint_as_float(hi);
            rest[frag_at(b + i, lane)] = __uint_as_float(lo);
          }
        }
      }
      round_end();
    }
  } else {
    // ---- P
    for (int r = -3; r <= chunks; ++r) {
      const int c = r;
      if (c >= 0 && c < chunks) {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          float acc[4][4];
          mul_keys(acc, sm.q[c % 3], sm.k[c & 3], sm.gh[c & 7], sm.gl[c & 7], i, lane);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j >= 2 * i + 2) break;
            uint32_t hi[4], lo[4];             // this lane's words of the operand tile
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int ri = 16 * i + (e >> 1) * 8 + g, cj = 8 * j + 2 * t + (e & 1);
              const int slot = (e >> 1) + 2 * (e & 1);
              const float p = acc[j][e] * scale;
              split_tf32(cj < ri ? p : 0.f, hi[slot], lo[slot]);
              if (cj == ri) sm.pd[c & 1][ri] = p;
            }
            *reinterpret_cast<uint4*>(&sm.p[c & 1][0][4 * i + j][lane * 4]) =
                make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(&sm.p[c & 1][1][4 * i + j][lane * 4]) =
                make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        }
      }
      round_end();
    }
  }
}

}  // namespace pipe

int gdn_pipe_launch(const __half* qkv, int conv_dim, const float* ab, const float* a_log,
                    const float* dt_bias, const Segment* segs, int n_segs, const int* row_slot,
                    const int* row_pos, int hk, int hv, float* state, float* out,
                    cudaStream_t stream) {
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, pipe::gdn_pipe_kernel, sizeof(pipe::Smem))) return e;
  pipe::gdn_pipe_kernel<<<dim3(hv * 2, n_segs), pipe::THREADS, sizeof(pipe::Smem), stream>>>(
      qkv, conv_dim, ab, a_log, dt_bias, segs, row_slot, row_pos, hk, hv, state, out);
  return 0;
}

}  // namespace orinfer
