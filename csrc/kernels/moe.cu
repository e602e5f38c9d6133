// Mixture-of-experts routing and data movement: fused router projection + softmax + top-k,
// deterministic expert counts / offsets / tile table / slot assignment (counts by shared-memory
// atomics, whose order shows nowhere; slots in row order),
// dispatch of quantised rows into expert-contiguous slots, and the weighted combine.
// Replaces router_projection / router_topk (kernels/cuda/model/moe.py:16,413),
// expert_histogram* / expert_offsets / expert_tiles (moe.py:177-286,558-713),
// expert_dispatch (moe.py:286) and moe_combine (moe.py:498-557) of the reference.
#include <cooperative_groups.h>

#include "api.h"
#include "common.cuh"
#include "tp_comm.cuh"

namespace cg = cooperative_groups;

namespace orinfer {

// ---------------------------------------------------------------- router + top-k
// logits[e] = x[row] . W[e] (fp16 inputs, fp32 accumulate); softmax over the first `experts`
// rows of W; top-k by repeated argmax with ties going to the lower expert id; optional
// renormalisation; row `experts` of W (when present) is the shared-expert gate, returned as
// sigmoid(logit).

// Softmax statistics and top-k of one row by one warp; `logits` [experts (+ 1)] in shared
// memory, overwritten.
__device__ __forceinline__ void topk_row(float* logits, int row, int experts, int has_shared,
                                         int top_k, int renorm, int* __restrict__ ids,
                                         float* __restrict__ probs,
                                         float* __restrict__ shared_gate) {
  const int lane = threadIdx.x & 31;
  float mx = -INFINITY;
  for (int e = lane; e < experts; e += 32) mx = fmaxf(mx, logits[e]);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int e = lane; e < experts; e += 32) sum += expf(logits[e] - mx);
  sum = warp_sum(sum);
  // Every lane keeps the best of its own logits and looks for another only when that one is taken;
  // lane k holds the k-th choice (the first 32; later ones go through memory).
  float best = -INFINITY;
  int bidx = 0x7fffffff;
  auto scan = [&]() {
    best = -INFINITY;
    bidx = 0x7fffffff;
    for (int e = lane; e < experts; e += 32) {
      const float v = logits[e];
      if (v > best) { best = v; bidx = e; }           // ascending e: first maximum wins
    }
  };
  scan();
  float chosen_sum = 0.f, my_prob = 0.f;
  int my_id = 0;
  for (int k = 0; k < top_k; ++k) {
    float top = best;
    int at = bidx;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, top, o);
      const int oi = __shfl_xor_sync(0xffffffffu, at, o);
      if (ov > top || (ov == top && oi < at)) { top = ov; at = oi; }
    }
    if (at >= experts) at = k;                      // no comparable logit left (NaN): any valid id
    const float p = expf(top - mx) / sum;
    chosen_sum += p;
    if (k < 32) {
      if (lane == k) {
        my_id = at;
        my_prob = p;
      }
    } else if (lane == 0) {
      ids[row * top_k + k] = at;
      probs[row * top_k + k] = p;
    }
    if ((at & 31) == lane) {
      logits[at] = -INFINITY;
      scan();
    }
  }
  if (lane < top_k) {
    ids[row * top_k + lane] = my_id;
    probs[row * top_k + lane] = renorm ? my_prob / chosen_sum : my_prob;
  }
  if (renorm && lane == 0)
    for (int k = 32; k < top_k; ++k) probs[row * top_k + k] /= chosen_sum;
  if (has_shared && lane == 0)
    shared_gate[row] = 1.f / (1.f + expf(-logits[experts]));
}

// General form: one CTA per token row, one warp per expert at a time.
__global__ void __launch_bounds__(256) router_topk_kernel(
    const __half* x, const __half* w, int hidden, int experts, int has_shared, int top_k,
    int renorm, int* __restrict__ ids, float* __restrict__ probs, float* __restrict__ shared_gate) {
  extern __shared__ float logits[];                 // [experts + 1]
  grid_wait();
  grid_release();
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = blockDim.x >> 5, total = experts + (has_shared ? 1 : 0);
  const __half* xr = x + static_cast<size_t>(row) * hidden;
  for (int e = warp; e < total; e += nw) {
    const __half* wr = w + static_cast<size_t>(e) * hidden;
    float acc = 0.f;
    for (int i = lane * 8; i < hidden; i += 256) {
      const int4 xa = *reinterpret_cast<const int4*>(xr + i);
      const int4 wa = *reinterpret_cast<const int4*>(wr + i);
      const __half2* xh = reinterpret_cast<const __half2*>(&xa);
      const __half2* wh = reinterpret_cast<const __half2*>(&wa);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 a = __half22float2(xh[j]), b = __half22float2(wh[j]);
        acc = fmaf(a.x, b.x, acc);
        acc = fmaf(a.y, b.y, acc);
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) logits[e] = acc;
  }
  __syncthreads();
  if (warp != 0) return;
  topk_row(logits, row, experts, has_shared, top_k, renorm, ids, probs, shared_gate);
}

// Tensor-core form (hidden % 256 == 0, at most 64 MAXT expert rows).  The general form
// streams the whole router matrix (0.5 to 2 MB) through every CTA, once per token row.  Here a
// cluster of eight CTAs takes 16 rows: CTA c owns an eighth of the 8-expert tiles, its WARPS
// warps a WARPS-th of the hidden channels each, and each CTA collects the logits of its share of
// the rows over distributed shared memory for the top-k.  Lane (g, t) loads 16 bytes of row g:
// the halves 4s..4s+3 are its fragments of step s, in x and W alike.
// The tensor core sums 16 FP16 products at a time and cuts the sum off instead of rounding it, so
// every such sum starts at zero and is added in FP32, the warps' parts pairwise: probabilities of
// 256 experts under 4096 channels are within 1.9e-7 of exact (the general form 2.9e-7, sums chained
// through the tensor core 6.6e-7).  The order depends on the router alone, so a row's logits do not
// depend on the packet's other rows.
// 128 experts x 2048 channels: 16 rows 25.9 -> 9.5 us, 2048 rows 95 -> 48; one step per turn of the
// loop: two take 57 us at 2048 rows.

constexpr int ROUTER_CL = 8;

template <int MAXT, int WARPS>
__global__ void __cluster_dims__(ROUTER_CL, 1, 1) __launch_bounds__(WARPS * 32) router_mma_kernel(
    const __half* x, const __half* w, int rows, int hidden, int experts, int has_shared, int top_k,
    int renorm, int* __restrict__ ids, float* __restrict__ probs, float* __restrict__ shared_gate) {
  constexpr int CL = ROUTER_CL, ROWS = 16, COLS = MAXT * 8 + 1, OWN = ROWS / CL;
  extern __shared__ float router_smem[];
  float(*part)[ROWS][COLS] = reinterpret_cast<float(*)[ROWS][COLS]>(router_smem);
  float* logits = router_smem + WARPS * ROWS * COLS;              // [OWN][total]
  grid_wait();
  grid_release();
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = static_cast<int>(cluster.block_rank());
  const int row0 = static_cast<int>(blockIdx.x) / CL * ROWS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int total = experts + (has_shared ? 1 : 0), tiles = (total + 7) / 8;
  const int t_lo = tiles * crank / CL, nt = tiles * (crank + 1) / CL - t_lo;
  float acc[MAXT][4];
#pragma unroll
  for (int i = 0; i < MAXT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  // rows past the last token or expert read the last one; their sums are not used
  const __half* xa = x + static_cast<size_t>(min(row0 + g, rows - 1)) * hidden + t * 8;
  const __half* xb = x + static_cast<size_t>(min(row0 + g + 8, rows - 1)) * hidden + t * 8;
  const int k_lo = hidden / WARPS * warp, k_hi = k_lo + hidden / WARPS;
#pragma unroll 1
  for (int k = k_lo; k < k_hi; k += 32) {
    const uint4 a = *reinterpret_cast<const uint4*>(xa + k);
    const uint4 b = *reinterpret_cast<const uint4*>(xb + k);
    uint4 wv[MAXT];
#pragma unroll
    for (int i = 0; i < MAXT; ++i)
      if (i < nt) {
        const int e = min((t_lo + i) * 8 + g, total - 1);
        const __half* we = w + static_cast<size_t>(e) * hidden + t * 8 + k;
        wv[i] = *reinterpret_cast<const uint4*>(we);
      }
#pragma unroll
    for (int i = 0; i < MAXT; ++i)
      if (i < nt) {
        float d[4] = {0.f, 0.f, 0.f, 0.f}, f[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(d, a.x, b.x, a.y, b.y, wv[i].x, wv[i].y);
        mma16816(f, a.z, b.z, a.w, b.w, wv[i].z, wv[i].w);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += d[j] + f[j];
      }
  }
#pragma unroll
  for (int i = 0; i < MAXT; ++i)
    if (i < nt)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        part[warp][g + (e >> 1) * 8][i * 8 + 2 * t + (e & 1)] = acc[i][e];
  cluster.sync();                                   // every CTA of the cluster runs
  for (int i = threadIdx.x; i < ROWS * nt * 8; i += WARPS * 32) {
    const int r = i / (nt * 8), c = i % (nt * 8), e = t_lo * 8 + c;
    float v[WARPS];
#pragma unroll
    for (int q = 0; q < WARPS; ++q) v[q] = part[q][r][c];
#pragma unroll
    for (int n = WARPS / 2; n > 0; n /= 2)
#pragma unroll
      for (int q = 0; q < n; ++q) v[q] += v[q + n];
    if (e < total) cluster.map_shared_rank(logits, r / OWN)[(r % OWN) * total + e] = v[0];
  }
  cluster.sync();
  const int row = row0 + crank * OWN + warp;
  if (warp < OWN && row < rows)
    topk_row(logits + warp * total, row, experts, has_shared, top_k, renorm, ids, probs,
             shared_gate);
}

template <int MAXT, int WARPS>
static int launch_router(const __half* x, const __half* w, int rows, int hidden, int experts,
                         int has_shared, int top_k, int renorm, int* ids, float* probs,
                         float* shared_gate, cudaStream_t stream) {
  const int total = experts + (has_shared ? 1 : 0);
  constexpr int PART = WARPS * 16 * (MAXT * 8 + 1);
  const size_t smem = (PART + 2 * static_cast<size_t>(total)) * sizeof(float);
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, router_mma_kernel<MAXT, WARPS>,
                                       (PART + 2 * 8 * ROUTER_CL * MAXT) * sizeof(float)))
    return e;
  const int grid = (rows + 15) / 16 * ROUTER_CL;
  launch_early(router_mma_kernel<MAXT, WARPS>, grid, WARPS * 32, smem, stream, x, w, rows, hidden,
               experts, has_shared, top_k, renorm, ids, probs, shared_gate);
  return static_cast<int>(cudaGetLastError());
}

// The same product for many rows (at most 136 expert rows, hidden / CL 384 or 512 channels).
// The form above reads a row eight times and the matrix once per 16 rows, in 64-byte pieces: 128 MB
// from L2 for 2048 rows.  Here a cluster of CL CTAs takes 64 rows and each of them a CL-th of the
// channels, copied to shared memory once (192 KB); eight warps hold 32 rows x a quarter of the
// expert tiles each, and the CTAs add up each other's parts for 64 / CL rows of the top-k.  Sums as
// above: 16 products in the tensor core, pairs of those added in FP32 in two alternating sums per
// CTA (probabilities of 128 experts: 1.18e-7 from exact at 2048 channels, 1.50e-7 at 4096; above
// 1.18e-7 and 1.62e-7).  At most 136 expert rows and 512 channels a CTA fit its shared memory; at
// least 384 channels, because the parts of 136 experts take the place of the 64 rows.  128 experts
// x 2048 channels, 2048 rows: 46.4 -> 19.8 us, 1024 rows 27.2 -> 19.5, 512 rows 22.8 -> 19.5; fewer
// rows are one wave of the form above (384: 10.1 us).  Half of it is the top-k, two rows per warp:
// with choices kept in memory and renormalised there it took 15 us more.
constexpr int ROUTER_ROWS = 64, ROUTER_TILES = 17, ROUTER_MANY = 512;

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p))
               : "memory");
}

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(256, 1) router_rows_kernel(
    const __half* x, const __half* w, int rows, int hidden, int experts, int has_shared, int top_k,
    int renorm, int* __restrict__ ids, float* __restrict__ probs, float* __restrict__ shared_gate) {
  constexpr int ROWS = ROUTER_ROWS, OWN = ROWS / CL, PER = (ROUTER_TILES + 3) / 4;
  extern __shared__ __align__(16) unsigned char router_raw[];
  const int total = experts + (has_shared ? 1 : 0), tiles = (total + 7) / 8;
  const int span = hidden / CL, pitch = span + 8;           // halves; rows 16 bytes apart in banks
  __half* xs = reinterpret_cast<__half*>(router_raw);       // [ROWS][pitch]
  __half* ws = xs + ROWS * pitch;                           // [8 tiles][pitch]
  grid_wait();
  grid_release();
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = static_cast<int>(cluster.block_rank());
  const int row0 = static_cast<int>(blockIdx.x) / CL * ROWS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int slabs = span / 128;
  for (int s = 0; s < slabs; ++s) {
    // rows past the last token or expert are copies of the last one; their sums are not used
    for (int i = tid; i < (ROWS + tiles * 8) * 16; i += 256) {
      const int r = i >> 4, c = s * 128 + (i & 15) * 8;
      const __half* src =
          r < ROWS ? x + static_cast<size_t>(min(row0 + r, rows - 1)) * hidden
                   : w + static_cast<size_t>(min(r - ROWS, total - 1)) * hidden;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(xs + r * pitch + c)),
                   "l"(src + crank * span + c)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int m0 = (warp & 1) * 32, first = warp >> 1;        // expert tiles first, first + 4, ...
  float acc[2][2][PER][4] = {};                             // [alternating sum][16 rows][tile]
  for (int s = 0; s < slabs; ++s) {
    // the copies of slab s have landed when at most slabs - 1 - s groups are under way
    if (s + 1 >= slabs) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else if (s + 2 >= slabs) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else if (s + 3 >= slabs) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else asm volatile("cp.async.wait_group 3;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int k = s * 128 + kk * 32;
      uint32_t a[2][2][4];                                  // [16 rows][16 channels]
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          ldmatrix4(a[m][h],
                    xs + (m0 + m * 16 + (lane & 15)) * pitch + k + h * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int tile = first + i * 4;
        if (tile >= tiles) break;
        uint32_t b[4];
        ldmatrix4(b, ws + (tile * 8 + (lane & 7)) * pitch + k + (lane >> 3) * 8);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          float d[4] = {0.f, 0.f, 0.f, 0.f}, f[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816(d, a[m][0][0], a[m][0][1], a[m][0][2], a[m][0][3], b[0], b[1]);
          mma16816(f, a[m][1][0], a[m][1][1], a[m][1][2], a[m][1][3], b[2], b[3]);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[kk & 1][m][i][e] += d[e] + f[e];
        }
      }
    }
  }
  __syncthreads();                                          // xs becomes the parts' buffer
  float* part = reinterpret_cast<float*>(xs);               // [ROWS][cols]
  const int cols = tiles * 8 + 1;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int tile = first + i * 4;
    if (tile >= tiles) break;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        part[(m0 + m * 16 + g + (e >> 1) * 8) * cols + tile * 8 + 2 * t + (e & 1)] =
            acc[0][m][i][e] + acc[1][m][i][e];
  }
  cluster.sync();
  float* logits = reinterpret_cast<float*>(ws);             // [OWN][total]
  for (int i = tid; i < OWN * total; i += 256) {
    const int r = i / total, e = i - r * total;
    float v[CL];
#pragma unroll
    for (int q = 0; q < CL; ++q)
      v[q] = cluster.map_shared_rank(part, q)[(crank * OWN + r) * cols + e];
#pragma unroll
    for (int n = CL / 2; n > 0; n /= 2)
#pragma unroll
      for (int q = 0; q < n; ++q) v[q] += v[q + n];
    logits[i] = v[0];
  }
  cluster.sync();                                           // nobody leaves while it is read
  for (int r = warp; r < OWN; r += 8) {
    const int row = row0 + crank * OWN + r;
    if (row < rows)
      topk_row(logits + r * total, row, experts, has_shared, top_k, renorm, ids, probs,
               shared_gate);
  }
}

inline size_t router_rows_smem(int hidden, int total, int cl) {
  return static_cast<size_t>(ROUTER_ROWS + (total + 7) / 8 * 8) * (hidden / cl + 8) * 2;
}

template <int CL>
static int launch_router_rows(const __half* x, const __half* w, int rows, int hidden, int experts,
                              int has_shared, int top_k, int renorm, int* ids, float* probs,
                              float* shared_gate, cudaStream_t stream) {
  static const int slot = runtime_new_slot();
  if (const int e = runtime_allow_smem(slot, router_rows_kernel<CL>, 220 * 1024)) return e;
  const int grid = (rows + ROUTER_ROWS - 1) / ROUTER_ROWS * CL;
  launch_early(router_rows_kernel<CL>, grid, 256,
               router_rows_smem(hidden, experts + (has_shared ? 1 : 0), CL), stream, x, w, rows,
               hidden, experts, has_shared, top_k, renorm, ids, probs, shared_gate);
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------- slots
// One CTA per local expert, one launch for everything the grouped GEMM needs to know: each CTA
// counts the assignments of all experts in shared memory (integers: the order does not
// matter), sums the counts and 128-row tiles before its own expert, writes its offset, count
// and tile-table entries, and numbers its own assignments in (row, k) order: slot[i] =
// offset[e] + rank of i among the assignments of e.  Under expert parallelism a rank owns
// experts [base_expert, base_expert + gridDim.x): ids outside that range get slot -1 (CTA 0
// writes those) and the combine skips them.
// More threads where there are many assignments to walk (16384 of them: 26 us with 256).
template <int THREADS>
__global__ void __launch_bounds__(THREADS) moe_plan_kernel(
    const int* ids, int assigns, int base_expert, int* counts, int* offsets, int* tiles, int* meta,
    int max_tiles, int* slots) {
  extern __shared__ int hist[];                     // [experts]
  constexpr int WARPS = THREADS / 32;
  __shared__ int red[2][WARPS], warp_count[WARPS];
  const int e = blockIdx.x, experts = gridDim.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  grid_wait();
  grid_release();
  for (int i = tid; i < experts; i += THREADS) hist[i] = 0;
  __syncthreads();
  // a warp walks one contiguous run of assignments, 32 at a time
  const int steps = (assigns + THREADS - 1) / THREADS, lo = warp * steps * 32;
  int mine = 0;
#pragma unroll 4
  for (int s = 0; s < steps; ++s) {
    const int i = lo + s * 32 + lane;
    const int id = i < assigns ? ids[i] - base_expert : -1;
    if (id >= 0 && id < experts) atomicAdd(&hist[id], 1);
    mine += id == e;
    if (e == 0 && i < assigns && (id < 0 || id >= experts)) slots[i] = -1;
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) warp_count[warp] = mine;
  __syncthreads();
  int rows_before = 0, tiles_before = 0;
  for (int i = tid; i < e; i += THREADS) {
    rows_before += hist[i];
    tiles_before += (hist[i] + 127) / 128;
  }
  rows_before = __reduce_add_sync(0xffffffffu, rows_before);
  tiles_before = __reduce_add_sync(0xffffffffu, tiles_before);
  if (lane == 0) {
    red[0][warp] = rows_before;
    red[1][warp] = tiles_before;
  }
  __syncthreads();
  int off = 0, tile0 = 0, slot = 0;
#pragma unroll
  for (int q = 0; q < WARPS; ++q) {
    off += red[0][q];
    tile0 += red[1][q];
    if (q < warp) slot += warp_count[q];
  }
  const int count = hist[e], own_tiles = (count + 127) / 128;
  for (int j = tid; j < own_tiles; j += THREADS)
    if (tile0 + j < max_tiles) {
      int* entry = tiles + static_cast<size_t>(tile0 + j) * 4;
      entry[0] = e;
      entry[1] = off + j * 128;
      entry[2] = min(128, count - j * 128);
      entry[3] = j;
    }
  if (tid == 0) {
    counts[e] = count;
    offsets[e] = off;
    if (e == experts - 1) {
      offsets[experts] = off + count;
      meta[0] = min(tile0 + own_tiles, max_tiles);
    }
  }
  if (warp_count[warp] == 0) return;
  slot += off;
  for (int s = 0; s < steps; ++s) {
    const int i = lo + s * 32 + lane;
    const bool hit = i < assigns && ids[i] - base_expert == e;
    const unsigned ballot = __ballot_sync(0xffffffffu, hit);
    if (hit) slots[i] = slot + __popc(ballot & ((1u << lane) - 1u));
    slot += __popc(ballot);
  }
}

// Copies row blockIdx.x (INT8 values and scale) into the slots of its assignments: the row is
// read once and written top_k times in whole lines.  SPARSE (one slot a row): most rows may be free
// entries of a receive buffer, which are not read (131072 entries, 100 in use, 128 -> 105 us of
// which most is the numbering; all in use 159 -> 174).  With several slots a row, few rows of a
// rank go nowhere, and looking first costs 0.2 to 0.5 us of 4 to 7.
template <bool SPARSE>
__global__ void __launch_bounds__(128) moe_scatter_kernel(
    const int* slots, int top_k, const int8_t* q8, const float* scale, int K,
    int8_t* __restrict__ q8_sorted, float* __restrict__ scale_sorted) {
  grid_wait();
  grid_release();
  const int row = blockIdx.x;
  const int* sl = slots + static_cast<size_t>(row) * top_k;
  if (SPARSE && *sl < 0) return;
  const float s = scale[row];
  for (int j = threadIdx.x; j < top_k; j += blockDim.x)
    if (sl[j] >= 0) scale_sorted[sl[j]] = s;
  for (int c = threadIdx.x; c < K / 16; c += blockDim.x) {
    const int4 v = reinterpret_cast<const int4*>(q8 + static_cast<size_t>(row) * K)[c];
    for (int j = 0; j < top_k; ++j) {
      const int slot = sl[j];
      if (slot >= 0) reinterpret_cast<int4*>(q8_sorted + static_cast<size_t>(slot) * K)[c] = v;
    }
  }
}

// out[row] = fp16( sum_k prob[row,k] * expert_out[slot(row,k)] + gate[row] * shared[row] )
__global__ void __launch_bounds__(256) moe_combine_kernel(
    const __half* expert_out, const int* slots, const float* probs, int top_k,
    const __half* shared_out, const float* shared_gate, __half* __restrict__ out, int hidden,
    const PeerOut peers) {
  grid_wait();
  grid_release();
  const int row = blockIdx.x;
  for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    // four expert rows in flight at a time; a slot of another rank counts as weight zero
    for (int k0 = 0; k0 < top_k; k0 += 4) {
      float p[4];
      int4 raw[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = k0 + q, slot = k < top_k ? slots[row * top_k + k] : -1;
        p[q] = slot >= 0 ? probs[row * top_k + k] : 0.f;
        raw[q] = slot >= 0 ? *reinterpret_cast<const int4*>(
                                 expert_out + static_cast<size_t>(slot) * hidden + i)
                           : make_int4(0, 0, 0, 0);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const __half* h = reinterpret_cast<const __half*>(&raw[q]);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = fmaf(p[q], __half2float(h[j]), acc[j]);
      }
    }
    if (shared_out != nullptr) {
      const float g = shared_gate[row];
      const int4 raw =
          *reinterpret_cast<const int4*>(shared_out + static_cast<size_t>(row) * hidden + i);
      const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = fmaf(g, __half2float(h[j]), acc[j]);
    }
    __align__(16) __half o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = __float2half_rn(acc[j]);
    if (peers.tp == 0) {
      *reinterpret_cast<int4*>(out + static_cast<size_t>(row) * hidden + i) =
          *reinterpret_cast<const int4*>(o);
    } else {
      // expert-parallel combine: this rank's partial row goes straight into slot [rank] of
      // every rank's inbox; the consumer norm kernel sums the tp partials
      const size_t off = (static_cast<size_t>(peers.rank) * peers.rows_cap + row) * hidden + i;
      for (int d = 0; d < peers.tp; ++d)
        *reinterpret_cast<int4*>(peers.inbox[d] + off) = *reinterpret_cast<const int4*>(o);
    }
  }
  if (peers.tp != 0) peer_signal_done(peers, gridDim.x);
}

static int launch_dispatch(const int* ids, int rows, int top_k, int base_expert, int experts,
                           const int8_t* q8, const float* scale, int K, int* counts, int* offsets,
                           int* tiles, int* meta, int max_tiles, int* slots, int8_t* q8_sorted,
                           float* scale_sorted, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(experts) * sizeof(int);
  auto kernel = rows * top_k >= 4096 ? moe_plan_kernel<1024> : moe_plan_kernel<256>;
  if (smem > 48 * 1024) {                           // more than 12 288 experts on one rank
    const cudaError_t e = cudaFuncSetAttribute(
        kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  launch_early(kernel, experts, rows * top_k >= 4096 ? 1024 : 256, smem, stream, ids,
               rows * top_k, base_expert, counts, offsets, tiles, meta, max_tiles, slots);
  if (q8 != nullptr)                                // nullptr: only the slot numbering is wanted
    launch_early(top_k == 1 ? moe_scatter_kernel<true> : moe_scatter_kernel<false>, rows, 128, 0,
                 stream, slots, top_k, q8, scale, K, q8_sorted, scale_sorted);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace orinfer

using namespace orinfer;

// The router's form: rows per CTA or cluster.
static int router_form(int rows, int hidden, int total) {
  // Few experts leave most of a cluster's CTAs without a tile, and its two exchanges cost more than
  // reading a small matrix per row: 8 experts x 2048 channels, 16 rows, 4.6 us in the general
  // form against 6.3, 2048 rows 13.6 against 17.7; 16 experts 5.9 against 6.6; but 16 x 4096 11.0
  // against 9.2 and 24 x 2048 8.1 against 7.4.  Up to 32 x 2048 the general form is also ahead
  // where the clusters need one more wave than its CTAs (24 x 2048: 512 rows 8.7 against 9.8 us,
  // 768 rows 11.1 against 12.1, 1024 rows 18.0 against 12.6, 1536 rows 19.7 against 21.5).
  const int cells = total * hidden;
  const bool few = (total <= 17 && cells <= 17 * 2048) ||
                   (cells <= 32 * 2048 &&
                    ((rows >= 256 && rows <= 640) || (rows > 1100 && rows < 1900)));
  const int cl = hidden <= 2048 ? 4 : 8;
  if (!few && rows >= ROUTER_MANY && hidden % (cl * 128) == 0 && hidden / cl >= 384 &&
      hidden / cl <= 512 && total <= ROUTER_TILES * 8 &&
      router_rows_smem(hidden, total, cl) <= 220 * 1024)
    return ROUTER_ROWS;
  return !few && hidden % 256 == 0 && total <= 8 * 8 * 9 ? 16 : 1;
}

extern "C" {

int orinfer_router_form(int rows, int hidden, int experts, int has_shared) {
  return router_form(rows, hidden, experts + (has_shared ? 1 : 0));
}

int orinfer_router_topk(const __half* x, const __half* w, int rows, int hidden, int experts,
                        int has_shared, int top_k, int renorm, int* ids, float* probs,
                        float* shared_gate, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hidden % 8 || top_k < 1 || top_k > experts || experts > 4096) return -1;
  const int total = experts + (has_shared ? 1 : 0);
  const int form = runtime_ensure_init() == cudaSuccess ? router_form(rows, hidden, total) : 1;
  if (form == ROUTER_ROWS)
    return (hidden <= 2048 ? launch_router_rows<4> : launch_router_rows<8>)(
        x, w, rows, hidden, experts, has_shared, top_k, renorm, ids, probs, shared_gate, stream);
  if (form == 16) {
    // Wide routers read their matrix from few SMs in a decode step: more warps, more loads in
    // flight (16 rows, 512 experts: 26 -> 16 us).
#define ORINFER_ROUTER(MAXT, WARPS)                                                  \
  return launch_router<MAXT, WARPS>(x, w, rows, hidden, experts, has_shared, top_k,  \
                                            renorm, ids, probs, shared_gate, stream)
    if (total > 8 * 8 * 3) {
      if (hidden % 512 == 0) ORINFER_ROUTER(9, 16);
      ORINFER_ROUTER(9, 8);
    }
    ORINFER_ROUTER(3, 8);
#undef ORINFER_ROUTER
  }
  launch_early(router_topk_kernel, rows, 256, (experts + 1) * sizeof(float), stream, x, w, hidden,
               experts, has_shared, top_k, renorm, ids, probs, shared_gate);
  return static_cast<int>(cudaGetLastError());
}

// counts [E], offsets [E+1], tiles int32 [max_tiles,4] = (expert, first slot, rows,
// number of the tile within its expert),
// meta[0] = tile count, slots [rows*top_k]; q8_sorted / scale_sorted get the dispatched rows.
int orinfer_moe_dispatch(const int* ids, int rows, int top_k, int experts, const int8_t* q8,
                         const float* scale, int K, int* counts, int* offsets, int* tiles,
                         int* meta, int max_tiles, int* slots, int8_t* q8_sorted,
                         float* scale_sorted, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (K % 16) return -1;
  return launch_dispatch(ids, rows, top_k, 0, experts, q8, scale, K, counts, offsets, tiles, meta,
                         max_tiles, slots, q8_sorted, scale_sorted, stream);
}

// Expert-parallel dispatch: this rank owns experts [base_expert, base_expert + local_experts);
// only rows routed there are counted and copied, every other slot is -1.
int orinfer_moe_dispatch_ep(const int* ids, int rows, int top_k, int base_expert,
                            int local_experts, const int8_t* q8, const float* scale, int K,
                            int* counts, int* offsets, int* tiles, int* meta, int max_tiles,
                            int* slots, int8_t* q8_sorted, float* scale_sorted,
                            cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (K % 16) return -1;
  return launch_dispatch(ids, rows, top_k, base_expert, local_experts, q8, scale, K, counts,
                         offsets, tiles, meta, max_tiles, slots, q8_sorted, scale_sorted, stream);
}

// Combine whose result rows are pushed into every rank's inbox (slot [rank]) over NVLink and
// signalled, instead of being written locally: the all-reduce of the expert-parallel partial
// sums is completed by the consumer norm kernel.
int orinfer_moe_combine_peer(const __half* expert_out, const int* slots, const float* probs,
                             int rows, int top_k, const __half* shared_out,
                             const float* shared_gate, const OrinferPeerOut* peers, int hidden,
                             cudaStream_t stream) {
  if (rows <= 0 || peers == nullptr) return -1;
  if (hidden % 8 || rows > peers->rows_cap) return -1;
  if (peers->tp < 1 || peers->tp > TP_MAX) return -1;
  PeerOut po;
  for (int i = 0; i < TP_MAX; ++i) {
    po.inbox[i] = reinterpret_cast<__half*>(peers->inbox[i]);
    po.flag[i] = peers->flag[i];
  }
  po.sent = peers->sent;
  po.ticket = peers->ticket;
  po.tp = peers->tp;
  po.rank = peers->rank;
  po.rows_cap = peers->rows_cap;
  po.rows_per = 0;
  moe_combine_kernel<<<rows, 256, 0, stream>>>(expert_out, slots, probs, top_k, shared_out,
                                               shared_gate, nullptr, hidden, po);
  return static_cast<int>(cudaGetLastError());
}

int orinfer_moe_combine(const __half* expert_out, const int* slots, const float* probs, int rows,
                        int top_k, const __half* shared_out, const float* shared_gate,
                        __half* out, int hidden, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hidden % 8) return -1;
  launch_early(moe_combine_kernel, rows, 256, 0, stream, expert_out, slots, probs, top_k,
               shared_out, shared_gate, out, hidden, PeerOut{});
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
