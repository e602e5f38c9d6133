// Gated-delta-rule linear attention kernels, natively batched over the requests of a packet
// through a segment table (first row, rows, state slot):
//   small_proj   : fp32 out[M,N] = x[M,H] . W[N,H]^T for narrow N (the a/b gate projection)
//   gdn_conv     : width-4 causal depthwise conv over q|k|v channels with a 3-row per-request
//                  history, SiLU, per-head L2 norm of q and k; then the history update
//   gdn_scan     : recurrence on the FP32 state, which lives in registers across a segment: row by
//                  row for short segments, in chunks of 32 rows (a triangular system and matrix
//                  products on the tensor cores) for long ones
//   gdn_gated_norm : per-head RMSNorm(o) * w * SiLU(z) (or sigmoid(z))
// Replace gdn_ab_tensorcore (kernels/cuda/operators/op07_gdn_ab.py:16), gdn_conv_prep
// (op08_gdn_conv_prep.py:23-278), gdn_gates (op09_gdn_gates.py:26-76), gdn_sequence
// (kernels/cuda/model/gdn_sequence.py:19-250) and gated_norm (op17_gdn_gated_norm.py:15-71).
#include "api.h"
#include "common.cuh"
#include "gdn_chunk.cuh"

namespace orinfer {

// ---------------------------------------------------------------- small projection
__global__ void __launch_bounds__(256) small_proj_kernel(
    const __half* x, const __half* w, float* __restrict__ out, int hidden, int n) {
  grid_wait();
  grid_release();
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __half* xr = x + static_cast<size_t>(row) * hidden;
  for (int e = warp; e < n; e += blockDim.x >> 5) {
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
    if (lane == 0) out[static_cast<size_t>(row) * n + e] = acc;
  }
}

// ---------------------------------------------------------------- conv + SiLU + L2 norm
// grid (rows, heads) with heads = 2*HK + HV of D channels each; block = D threads.
// x row layout: q | k | v | z  (z untouched).  hist: fp16 [slots, 3, conv_dim], oldest first.
template <int D>
__global__ void __launch_bounds__(D) gdn_conv_kernel(
    const __half* __restrict__ x, int x_stride, const __half* __restrict__ weight,
    const __half* __restrict__ hist, const int* __restrict__ row_first,
    const int* __restrict__ row_slot, const int* __restrict__ row_pos, int conv_dim,
    int qk_heads, __half* __restrict__ y) {
  const int row = blockIdx.x, head = blockIdx.y, c = head * D + threadIdx.x;
  const int first = row_first[row], slot = row_slot[row];
  const bool fresh = row_pos[first] == 0;
  const __half* wc = weight + static_cast<size_t>(c) * 4;
  float acc = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int src = row - 3 + j;                       // tap j reads the row 3-j steps back
    float v;
    if (src >= first) {
      v = __half2float(x[static_cast<size_t>(src) * x_stride + c]);
    } else {
      // rows before the chunk come from the history: index 3 - (first - src) from its end
      const int back = first - src;                    // 1..3
      v = fresh ? 0.f
                : __half2float(hist[(static_cast<size_t>(slot) * 3 + (3 - back)) * conv_dim + c]);
    }
    acc = fmaf(v, __half2float(wc[j]), acc);
  }
  float val = round_f16(acc * sigmoid_pair(make_float2(acc, acc)).x);
  if (head < qk_heads) {
    __shared__ float red[D / 32];
    float ss = warp_sum(val * val);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) tot += red[i];
    val = round_f16(val * rsqrtf(tot + 1e-6f));
  }
  y[static_cast<size_t>(row) * conv_dim + c] = __float2half_rn(val);
}

// The same convolution, eight channels per thread (16-byte loads and stores) over a strip of
// consecutive rows: the three earlier rows stay in registers as floats, so a packet's rows are read
// and converted once, and the arithmetic goes two channels to an instruction (sigmoid_pair).  A
// head is D / 8 neighbouring lanes.  Grid (strips, conv_dim / 2048), as many strips as fit the
// machine at once: what a strip costs ahead of its first row is paid by one wave of CTAs.  R = 1:
// strips of one row, for packets that have no more rows than that.
// 2100 rows x 8192 channels: 89 us a row at a time, 36 in strips of eight rows and 45 instructions
// a value, 27 now with 21 (68 MB; issue slots 50 %, the exponential and reciprocal unit 38 %,
// sixteen warps per SM); 64 rows 7.6 -> 6.8 us.
template <int D, int R>
__global__ void __launch_bounds__(256, 2) gdn_conv_vec_kernel(
    const __half* x, int x_stride, const __half* weight, const __half* hist, const int* row_first,
    const int* row_slot, const int* row_pos, int rows, int conv_dim, int qk_channels, int strip,
    __half* __restrict__ y) {
  constexpr int LANES = D / 8;
  grid_wait();
  grid_release();
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8, row0 = blockIdx.x * strip;
  const int end = min(rows, row0 + strip);
  if (row0 >= rows) return;
  if (c >= conv_dim) return;                       // whole heads, so whole lane groups
  const unsigned group = LANES == 32 ? 0xffffffffu
                                     : ((1u << LANES) - 1u) << (threadIdx.x & 31 & ~(LANES - 1));
  auto load = [&](int row) {
    return *reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * x_stride + c);
  };
  auto floats = [](float2 (&to)[4], const uint4& raw) {
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) to[i] = __half22float2(h[i]);
  };
  float2 w[4][4];                                  // [tap][pair of channels]
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 raw = reinterpret_cast<const uint4*>(weight + static_cast<size_t>(c) * 4)[i];
    const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j][i] = make_float2(__half2float(h[j]), __half2float(h[4 + j]));
  }
  // Row r is in win[r % 4] and comes R rows ahead of its use.  A strip that lies inside a run,
  // three rows from its first, needs nothing else.
  float2 win[4][4];
  uint4 next[R];
#pragma unroll
  for (int u = 0; u < R; ++u)
    if (row0 + u < end) next[u] = load(row0 + u);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int src = row0 - 3 + j;
    floats(win[j + 1], src >= 0 ? load(src) : make_uint4(0, 0, 0, 0));
  }
  const int first0 = row_first[row0];
  const bool inside = row0 - first0 >= 3 && row_first[end - 1] == first0;
  int row = row0;
  auto one_row = [&](int u) {                      // u = row % R
    floats(win[u], next[u]);
    if (row + R < end) next[u] = load(row + R);
    const int first = inside ? first0 : row_first[row];
    float2 acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = make_float2(0.f, 0.f);
    if (row - first < 3) {                         // rows before the run come from its history
      const bool fresh = row_pos[first] == 0;
      const int slot = row_slot[row];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int back = first - (row - 3 + j);    // 1..3 rows before the run
        float2 tap[4];
        if (back > 0) {
          const __half* kept = hist + (static_cast<size_t>(slot) * 3 + (3 - back)) * conv_dim + c;
          floats(tap, fresh ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4*>(kept));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) tap[i] = win[(u + 1 + j) & 3][i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = fma2(tap[i], w[j][i], acc[i]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = fma2(win[(u + 1 + j) & 3][i], w[j][i], acc[i]);
    }
    float ss = 0.f;
    uint4 packed;
    __half2* h = reinterpret_cast<__half2*>(&packed);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i] = fma2(win[u][i], w[3][i], acc[i]);
      acc[i] = mul2(acc[i], sigmoid_pair(acc[i]));
      h[i] = __floats2half2_rn(acc[i].x, acc[i].y);
    }
    if (c < qk_channels) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i] = __half22float2(h[i]);
        ss = fmaf(acc[i].x, acc[i].x, ss);
        ss = fmaf(acc[i].y, acc[i].y, ss);
      }
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) ss += __shfl_xor_sync(group, ss, o);
      const float inv = rsqrtf(ss + 1e-6f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 n = mul2(acc[i], make_float2(inv, inv));
        h[i] = __floats2half2_rn(n.x, n.y);
      }
    }
    *reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * conv_dim + c) = packed;
  };
  while (row < end) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
      if (row >= end) break;
      one_row(u);
      ++row;
    }
  }
}

// New history = last three pre-conv rows of (old history ++ chunk).  grid (segments, channel
// blocks); VEC channels per thread.  (One CTA per segment with 2-byte accesses took 21 us for
// 64 segments, this form 2.9 us.)
template <int VEC>
__global__ void __launch_bounds__(256) gdn_history_kernel(
    const __half* x, int x_stride, const Segment* segs, const int* row_slot, const int* row_pos,
    int conv_dim, __half* hist, const int* accepted) {
  grid_wait();
  grid_release();
  Segment s = segs[blockIdx.x];
  if (accepted != nullptr) {                 // commit of a verified prefix of the rows
    s.rows = min(accepted[blockIdx.x], s.rows);
  }
  if (s.rows <= 0) return;
  const int c = (blockIdx.y * 256 + threadIdx.x) * VEC;
  if (c >= conv_dim) return;
  struct __align__(VEC * 2) Chunk {
    __half h[VEC];
  };
  const bool fresh = row_pos[s.row_start] == 0;
  __half* h = hist + static_cast<size_t>(row_slot[s.row_start]) * 3 * conv_dim;
  Chunk v[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int idx = s.rows - 3 + j;          // index into the chunk, < 0 = history
    if (idx >= 0) {
      const __half* row = x + static_cast<size_t>(s.row_start + idx) * x_stride;
      v[j] = *reinterpret_cast<const Chunk*>(row + c);
    } else if (fresh) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[j].h[i] = __float2half(0.f);
    } else {
      v[j] = *reinterpret_cast<const Chunk*>(h + static_cast<size_t>(3 + idx) * conv_dim + c);
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
    *reinterpret_cast<Chunk*>(h + static_cast<size_t>(j) * conv_dim + c) = v[j];
}

// ---------------------------------------------------------------- sequential scan
// grid (HV * D/DC, segments); 256 threads.  The columns of the DxD state are independent in
// the recurrence, so a CTA owns DC value columns of one head: thread t owns column
// c0 + t % DC and key rows [ROWS*(t/DC), +ROWS), kept in registers for the whole segment.
// Launched with DC = D (one CTA per head): the state is read and written in whole rows by the
// fewest CTAs, which is what a decode step over many sequences is bound by.  The operands of
// step t+1 are fetched into registers while step t computes.  (Few segments: see
// gdn_scan_split_kernel below.)
template <int D, int DC>
__global__ void __launch_bounds__(256) gdn_scan_kernel(
    const __half* qkv, int conv_dim, const float* ab, const float* a_log, const float* dt_bias,
    const Segment* segs, const int* row_slot, const int* row_pos, int hk, int hv, float* state,
    float* __restrict__ out, float* __restrict__ factors, int long_rows) {
  // factors != nullptr: a verification pass.  The state is NOT written back; instead every
  // step records (decay, k[D], delta[D]) so that gdn_commit can replay exactly the accepted
  // prefix of the rows onto the stored state.
  constexpr int SPLIT = D / DC, PARTS = 256 / DC, ROWS = D / PARTS;
  static_assert(ROWS % 4 == 0, "four independent accumulators");
  grid_wait();
  grid_release();
  const int vh = blockIdx.x / SPLIT, c0 = (blockIdx.x % SPLIT) * DC;
  const Segment seg = segs[blockIdx.y];
  if (seg.rows <= 0 || seg.rows >= long_rows) return;  // long runs: gdn_chunk_kernel
  const int kh = vh / (hv / hk);
  const int dv = c0 + threadIdx.x % DC, part_id = threadIdx.x / DC;
  const int slot = row_slot[seg.row_start];
  const bool fresh = row_pos[seg.row_start] == 0;
  float* sp = state + ((static_cast<size_t>(slot) * hv + vh) * D + part_id * ROWS) * D + dv;
  float s[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) s[i] = fresh ? 0.f : sp[static_cast<size_t>(i) * D];
  __shared__ float ks[2][D], qs[2][D], part[PARTS][DC], opart[PARTS][DC];
  const float alog = expf(a_log[vh]), bias = dt_bias[vh];
  const float scale = rsqrtf(static_cast<float>(D));
  const int dk_total = hk * D;
  // which q/k element this thread stages (threads [0, D) -> q, [D, 2D) -> k)
  const bool is_q = threadIdx.x < D, is_k = !is_q && threadIdx.x < 2 * D;
  const int qk_col = is_q ? kh * D + threadIdx.x : dk_total + kh * D + threadIdx.x - D;
  const int v_col = 2 * dk_total + vh * D + dv;
  size_t row = static_cast<size_t>(seg.row_start);
  __half n_qk = (is_q || is_k) ? qkv[row * conv_dim + qk_col] : __float2half(0.f);
  __half n_v = qkv[row * conv_dim + v_col];
  float n_a = ab[row * 2 * hv + vh], n_b = ab[row * 2 * hv + hv + vh];
  for (int t = 0; t < seg.rows; ++t, ++row) {
    const int buf = t & 1;
    if (is_q) qs[buf][threadIdx.x] = __half2float(n_qk) * scale;
    if (is_k) ks[buf][threadIdx.x - D] = __half2float(n_qk);
    const float a = n_a, b = n_b, v = __half2float(n_v);
    if (t + 1 < seg.rows) {                            // operands of the next step, in flight
      const size_t nr = row + 1;
      if (is_q || is_k) n_qk = qkv[nr * conv_dim + qk_col];
      n_v = qkv[nr * conv_dim + v_col];
      n_a = ab[nr * 2 * hv + vh];
      n_b = ab[nr * 2 * hv + hv + vh];
    }
    __syncthreads();
    const float* kp = ks[buf] + part_id * ROWS;
    const float* qp = qs[buf] + part_id * ROWS;
    float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS; i += 4) {
      p0 = fmaf(s[i], kp[i], p0);
      p1 = fmaf(s[i + 1], kp[i + 1], p1);
      p2 = fmaf(s[i + 2], kp[i + 2], p2);
      p3 = fmaf(s[i + 3], kp[i + 3], p3);
    }
    const float xg = a + bias;
    const float softplus = xg > 20.f ? xg : log1pf(expf(xg));
    const float decay = expf(-alog * softplus);
    const float beta = __frcp_rn(1.f + expf(-b));
    part[part_id][threadIdx.x % DC] = ((p0 + p1) + (p2 + p3)) * decay;
    __syncthreads();
    float full = 0.f;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) full += part[i][threadIdx.x % DC];
    const float delta = beta * (v - full);
    if (factors != nullptr) {
      float* f = factors + (row * hv + vh) * (2 * D + 1);
      if (part_id == 0) f[1 + D + dv] = delta;
      if (c0 == 0) {
        if (threadIdx.x == 0) f[0] = decay;
        if (threadIdx.x < D) f[1 + threadIdx.x] = ks[buf][threadIdx.x];
      }
    }
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS; i += 4) {
      s[i] = fmaf(kp[i], delta, s[i] * decay);
      s[i + 1] = fmaf(kp[i + 1], delta, s[i + 1] * decay);
      s[i + 2] = fmaf(kp[i + 2], delta, s[i + 2] * decay);
      s[i + 3] = fmaf(kp[i + 3], delta, s[i + 3] * decay);
      o0 = fmaf(s[i], qp[i], o0);
      o1 = fmaf(s[i + 1], qp[i + 1], o1);
      o2 = fmaf(s[i + 2], qp[i + 2], o2);
      o3 = fmaf(s[i + 3], qp[i + 3], o3);
    }
    opart[part_id][threadIdx.x % DC] = (o0 + o1) + (o2 + o3);
    __syncthreads();
    if (part_id == 0) {
      float tot = 0.f;
#pragma unroll
      for (int i = 0; i < PARTS; ++i) tot += opart[i][threadIdx.x % DC];
      out[(row * hv + vh) * D + dv] = tot;
    }
  }
  if (factors == nullptr) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) sp[static_cast<size_t>(i) * D] = s[i];
  }
}

// ---------------------------------------------------------------- sequential scan, split heads
// The same recurrence for the case of few segments (prefill, small decode batches), where one
// CTA per head leaves most SMs idle and every step pays its own global-memory latency.
// grid (HV * D/32, segments): a CTA owns 32 value columns of one head.  Thread t owns column
// t / 8 and key rows [ROWS*(t % 8), +ROWS): the eight partial dot products of a column sit in
// neighbouring lanes and are combined with three shuffles, so a step needs no barrier.  q, k,
// v and the gates of the next SCAN_STEPS rows are staged in shared memory with cp.async while
// the current block computes; outputs leave in whole 128-byte rows once per block.
constexpr int SCAN_STEPS = 16;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}

template <int D>
__global__ void __launch_bounds__(256) gdn_scan_split_kernel(
    const __half* qkv, int conv_dim, const float* ab, const float* a_log, const float* dt_bias,
    const Segment* segs, const int* row_slot, const int* row_pos, int hk, int hv, float* state,
    float* __restrict__ out, float* __restrict__ factors, int long_rows) {
  constexpr int DC = 32, SPLIT = D / DC, PARTS = 8, ROWS = D / PARTS, T = SCAN_STEPS;
  constexpr int CH = D / 4 + DC / 8;                 // 16-byte units of one staged row
  grid_wait();
  grid_release();
  const int vh = blockIdx.x / SPLIT, c0 = (blockIdx.x % SPLIT) * DC;
  const Segment seg = segs[blockIdx.y];
  if (seg.rows <= 0 || seg.rows >= long_rows) return;  // long runs: gdn_chunk_kernel
  const int kh = vh / (hv / hk);
  const int col = threadIdx.x >> 3, part = threadIdx.x & 7;
  const int slot = row_slot[seg.row_start];
  const bool fresh = row_pos[seg.row_start] == 0;
  float* sp = state + ((static_cast<size_t>(slot) * hv + vh) * D + part * ROWS) * D + c0 + col;
  float s[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) s[i] = fresh ? 0.f : sp[static_cast<size_t>(i) * D];
  __shared__ __align__(16) __half qk_s[2][T][2 * D];
  __shared__ __align__(16) __half v_s[2][T][DC];
  __shared__ float dec_s[2][T], beta_s[2][T], o_s[T][DC];
  const float alog = expf(a_log[vh]), bias = dt_bias[vh];
  const float scale = rsqrtf(static_cast<float>(D));
  const int dk_total = hk * D;
  const int blocks = (seg.rows + T - 1) / T;

  auto stage = [&](int b) {
    const int n = min(T, seg.rows - b * T), buf = b & 1;
    for (int idx = threadIdx.x; idx < n * CH; idx += 256) {
      const int t = idx / CH, c = idx % CH;
      const __half* base = qkv + static_cast<size_t>(seg.row_start + b * T + t) * conv_dim;
      if (c < D / 8)
        cp_async16(&qk_s[buf][t][c * 8], base + kh * D + c * 8);
      else if (c < D / 4)
        cp_async16(&qk_s[buf][t][D + (c - D / 8) * 8], base + dk_total + kh * D + (c - D / 8) * 8);
      else
        cp_async16(&v_s[buf][t][(c - D / 4) * 8],
                   base + 2 * dk_total + vh * D + c0 + (c - D / 4) * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float n_a = 0.f, n_b = 0.f;
  auto gates = [&](int b) {                            // threads [0, T): gate inputs of block b
    const int t = b * T + threadIdx.x;
    if (threadIdx.x < T && t < seg.rows) {
      const size_t row = static_cast<size_t>(seg.row_start + t);
      n_a = ab[row * 2 * hv + vh];
      n_b = ab[row * 2 * hv + hv + vh];
    }
  };
  stage(0);
  gates(0);
  for (int b = 0; b < blocks; ++b) {
    const int buf = b & 1, n = min(T, seg.rows - b * T);
    if (threadIdx.x < T) {
      const float xg = n_a + bias;
      const float softplus = xg > 20.f ? xg : log1pf(expf(xg));
      dec_s[buf][threadIdx.x] = expf(-alog * softplus);
      beta_s[buf][threadIdx.x] = __frcp_rn(1.f + expf(-n_b));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                  // block b staged; everyone has left block b-1
    if (b + 1 < blocks) {
      stage(b + 1);
      gates(b + 1);
    }
    for (int t = 0; t < n; ++t) {
      const size_t row = static_cast<size_t>(seg.row_start + b * T + t);
      float kk[ROWS], qq[ROWS];
      const uint4* kp = reinterpret_cast<const uint4*>(&qk_s[buf][t][D + part * ROWS]);
      const uint4* qp = reinterpret_cast<const uint4*>(&qk_s[buf][t][part * ROWS]);
#pragma unroll
      for (int j = 0; j < ROWS / 8; ++j) {
        const uint4 kr = kp[j], qr = qp[j];
        const __half2* kh2 = reinterpret_cast<const __half2*>(&kr);
        const __half2* qh2 = reinterpret_cast<const __half2*>(&qr);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 kf = __half22float2(kh2[e]), qf = __half22float2(qh2[e]);
          kk[j * 8 + 2 * e] = kf.x;
          kk[j * 8 + 2 * e + 1] = kf.y;
          qq[j * 8 + 2 * e] = qf.x;
          qq[j * 8 + 2 * e + 1] = qf.y;
        }
      }
      float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
      for (int i = 0; i < ROWS; i += 4) {
        p0 = fmaf(s[i], kk[i], p0);
        p1 = fmaf(s[i + 1], kk[i + 1], p1);
        p2 = fmaf(s[i + 2], kk[i + 2], p2);
        p3 = fmaf(s[i + 3], kk[i + 3], p3);
      }
      float pred = (p0 + p1) + (p2 + p3);
      pred += __shfl_xor_sync(0xffffffffu, pred, 1);
      pred += __shfl_xor_sync(0xffffffffu, pred, 2);
      pred += __shfl_xor_sync(0xffffffffu, pred, 4);
      const float decay = dec_s[buf][t], beta = beta_s[buf][t];
      const float v = __half2float(v_s[buf][t][col]);
      const float delta = beta * (v - pred * decay);
      if (factors != nullptr) {
        float* f = factors + (row * hv + vh) * (2 * D + 1);
        if (part == 0) f[1 + D + c0 + col] = delta;
        if (c0 == 0) {
          if (threadIdx.x == 0) f[0] = decay;
          if (threadIdx.x < D) f[1 + threadIdx.x] = __half2float(qk_s[buf][t][D + threadIdx.x]);
        }
      }
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int i = 0; i < ROWS; i += 4) {
        s[i] = fmaf(kk[i], delta, s[i] * decay);
        s[i + 1] = fmaf(kk[i + 1], delta, s[i + 1] * decay);
        s[i + 2] = fmaf(kk[i + 2], delta, s[i + 2] * decay);
        s[i + 3] = fmaf(kk[i + 3], delta, s[i + 3] * decay);
        o0 = fmaf(s[i], qq[i], o0);
        o1 = fmaf(s[i + 1], qq[i + 1], o1);
        o2 = fmaf(s[i + 2], qq[i + 2], o2);
        o3 = fmaf(s[i + 3], qq[i + 3], o3);
      }
      float o = (o0 + o1) + (o2 + o3);
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      o += __shfl_xor_sync(0xffffffffu, o, 4);
      if (part == 0) o_s[t][col] = o * scale;
    }
    __syncthreads();                  // o_s complete (and re-used by the next block)
    for (int idx = threadIdx.x; idx < n * DC; idx += 256) {
      const int t = idx / DC, c = idx % DC;
      out[(static_cast<size_t>(seg.row_start + b * T + t) * hv + vh) * D + c0 + c] = o_s[t][c];
    }
  }
  if (factors == nullptr) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) sp[static_cast<size_t>(i) * D] = s[i];
  }
}

// ---------------------------------------------------------------- chunked form
// Long runs (prefill) in chunks of 32 rows: inside a chunk the recurrence is a triangular system
// and everything else is a matrix product, so a chunk costs a few thousand cycles instead of 32
// dependent steps.  With G_i the running sum of log decays inside the chunk and S the state
// before it,
//   A[i][j] = beta_i e^(G_i - G_j) k_i.k_j (j < i),   T = (I + A)^-1
//   Delta   = T B,  B_i = beta_i (v_i - e^G_i S^T k_i)
//   o_i     = e^G_i S^T q_i + sum_{j <= i} P[i][j] Delta_j,  P[i][j] = e^(G_i - G_j) q_i.k_j
//   S      <- e^G_32 S + sum_j k_j (x) e^(G_32 - G_j) Delta_j
// grid (2 HV, segments), six warps.  Warps 0..3 own 16 value channels each and keep their
// 16 x 128 slice of S^T in registers as MMA accumulators, whose layout is also that of an A
// operand: S^T K^T, B^T T^T, Delta^T P^T and Delta^T K chain through registers and no warp
// waits for another inside a chunk.  Warps 4 (A, T) and 5 (P) prepare the next chunk, which
// does not depend on the state, while the chunk after that is copied in.
//
// Precision: k, q and v are FP16 and enter products exactly.  FP32 operands are split: S into
// FP16 halves under a power-of-two scale per value channel, Delta for the state update into three
// FP16 parts, T and P off the diagonal into TF32 pairs; their diagonals, which carry most of the
// sums, are multiplied in FP32.  A tensor-core sum is cut off, not rounded, so each holds 32
// products at most and is added to the others by FP32 additions.  The G are summed in FP64 and
// subtracted as FP32 pairs, so that e^(G_i - G_j) keeps FP32 accuracy when |G| is large.
// Relative error against 64 bits, one run of 1050 rows: output 1.7e-7, state 1.1e-7 (the scan:
// 1.8e-7 and 1.3e-7; chained tensor-core sums of whole rows: 4.4e-7); with a memory of thousands
// of rows 2.0e-7 and 1.5e-7 (the scan, which rounds at every step: 1.9e-6 and 2.1e-6); with decays
// below 1/2 a row 1.6e-7 and 1.1e-7 (1.5e-7 and 1.1e-7).
//
// 32 heads of 128 channels, one run of 1050 rows: 406 us as a scan (0.39 us per dependent step),
// 195 us here (166 with chained sums), 164 since the helpers alone copy the chunks (two such runs,
// 128 CTAs, 190); 16 runs of 64 rows: 192 -> 84 -> 78 us.  Two CTAs per SM leave 168 registers and
// 168 bytes of spills a thread; issue slots 30 %, tensor pipe 24 %: dependent steps in few warps.
// Runs below GDN_LONG_ROWS keep the scan: one run of 36 rows takes 17.2 us there and 19.4 here, of
// 40 rows 19.4 both ways, of 63 rows 28.0 and 19.4 (two runs of 50: 33 and 20).  The scan's bits
// are those of a verification pass, whose segments are shorter.
constexpr int CHUNK_THREADS = 192;
struct ChunkSmem {
  __half k[3][CHUNK][136], q[3][CHUNK][136];   // rows padded to 17 16-byte units (ldmatrix)
  __half v[3][CHUNK][72];
  float t[2][CHUNK][40], p[2][CHUNK][40];      // T and P below the diagonal, row i, column j
  float pd[2][CHUNK];                          // diagonal of P (that of T is 1)
  float at[CHUNK][36];                         // A transposed: [j][i]
  float eg[2][CHUNK], beta[2][CHUNK], tail[2][CHUNK], total[2];
};

// FP16 head and remainder of two values (already scaled into the FP16 range)
__device__ __forceinline__ void split_half2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split_half3(float x, float y, uint32_t& hi, uint32_t& mid,
                                            uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  split_half2(x - f.x, y - f.y, mid, lo);
}
// D[i][0..7] (u-th group of eight columns) += X^T(16 x 32) M^T for a 32 x 32 matrix M in shared
// memory with zeros on and above the diagonal: X and M split into TF32 pairs.  A zero does not
// hide an infinity or a NaN of a later row in a tensor-core product, so a block on the diagonal
// whose rows hold one is summed term by term: earlier rows stay as they are.
__device__ __forceinline__ void mul_lower(float (&d)[4][4], const float (&x)[4][4],
                                          const float (*m)[40], int g, int t) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    uint32_t hi[4], lo[4];
    // k index t is row 8s + 2t of X, k index t + 4 is row 8s + 2t + 1
    split_tf32(x[s][0], hi[0], lo[0]);
    split_tf32(x[s][2], hi[1], lo[1]);
    split_tf32(x[s][1], hi[2], lo[2]);
    split_tf32(x[s][3], hi[3], lo[3]);
    const float size = (fabsf(x[s][0]) + fabsf(x[s][1])) + (fabsf(x[s][2]) + fabsf(x[s][3]));
    const bool wild = __any_sync(0xffffffffu, !(size < INFINITY));
    if (wild) {
#pragma unroll 1
      for (int src = 0; src < 4; ++src)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = 8 * s + 2 * src + e, from = (threadIdx.x & 28) | src;
          const float xa = __shfl_sync(0xffffffffu, x[s][e], from);
          const float xb = __shfl_sync(0xffffffffu, x[s][2 + e], from);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int i = 8 * s + 2 * t + c;
            if (j >= i) continue;
            d[s][c] = fmaf(xa, m[i][j], d[s][c]);
            d[s][2 + c] = fmaf(xb, m[i][j], d[s][2 + c]);
          }
        }
    }
#pragma unroll
    for (int u = s; u < 4; ++u) {
      if (u == s && wild) continue;
      const float2 b = *reinterpret_cast<const float2*>(&m[8 * u + g][8 * s + 2 * t]);
      uint32_t bh0, bl0, bh1, bl1;
      split_tf32(b.x, bh0, bl0);
      split_tf32(b.y, bh1, bl1);
      float part[4] = {0.f, 0.f, 0.f, 0.f};
      mma_tf32(part, hi, bl0, bl1);
      mma_tf32(part, lo, bh0, bh1);
      mma_tf32(part, hi, bh0, bh1);
#pragma unroll
      for (int e = 0; e < 4; ++e) d[u][e] += part[e];
    }
  }
}

__global__ void __launch_bounds__(CHUNK_THREADS, 2) gdn_chunk_kernel(
    const __half* __restrict__ qkv, int conv_dim, const float* __restrict__ ab,
    const float* __restrict__ a_log, const float* __restrict__ dt_bias,
    const Segment* __restrict__ segs, const int* __restrict__ row_slot,
    const int* __restrict__ row_pos, int hk, int hv, float* __restrict__ state,
    float* __restrict__ out) {
  constexpr int D = 128;
  extern __shared__ __align__(16) unsigned char chunk_smem[];
  ChunkSmem& sm = *reinterpret_cast<ChunkSmem*>(chunk_smem);
  grid_wait();
  grid_release();
  const Segment seg = segs[blockIdx.y];
  if (seg.rows < GDN_LONG_ROWS) return;
  const int vh = blockIdx.x >> 1, kh = vh / (hv / hk), dk_total = hk * D;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int mat = lane >> 3, mrow = lane & 7;          // this lane's row in an ldmatrix
  const int dv0 = (blockIdx.x & 1) * 64;
  const int chunks = (seg.rows + CHUNK - 1) / CHUNK;
  const float scale = rsqrtf(static_cast<float>(D));

  // Copy of one chunk by the two helper warps, eight threads a row, five 16-byte units each; rows
  // past the run become zeros.  (Spread over all threads, the copies held up the warps that carry
  // the state.)
  auto stage = [&](int c) {
    const int st = c % 3, n = min(CHUNK, seg.rows - c * CHUNK);
    const int at = (tid - 128) >> 3, s = (tid & 7) * 8;
#pragma unroll
    for (int pass = 0; pass < CHUNK / 8; ++pass) {
      const int r = pass * 8 + at, bytes = r < n ? 16 : 0;
      const __half* row =
          qkv + static_cast<size_t>(seg.row_start + c * CHUNK + min(r, n - 1)) * conv_dim + s;
      auto copy = [&](__half* dst, const __half* src) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src),
                     "r"(bytes)
                     : "memory");
      };
      copy(&sm.q[st][r][s], row + kh * D);
      copy(&sm.q[st][r][s + 64], row + kh * D + 64);
      copy(&sm.k[st][r][s], row + dk_total + kh * D);
      copy(&sm.k[st][r][s + 64], row + dk_total + kh * D + 64);
      copy(&sm.v[st][r][s], row + 2 * dk_total + vh * D + dv0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // ---- helpers: everything of chunk c that does not depend on the state
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
  auto prepare = [&](int c) {
    const int st = c % 3, buf = c & 1, helper = warp - 4;
    const bool live = c * CHUNK + lane < seg.rows;
    const float xg = n_a + bias;
    const float softplus = xg > 20.f ? xg : log1pf(expf(xg));
    // a decay that is zero in FP32 ends what a value was, also as the exponential of an infinity:
    // kept finite, so that differences of the sums stay defined (a NaN stays one)
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
    if (helper == 0) {
      sm.eg[buf][lane] = exp_pair(big_g);
      sm.beta[buf][lane] = beta;
      sm.tail[buf][lane] = exp_pair(last - big_g);
      if (lane == 0) sm.total[buf] = exp_pair(last);
    }
    // G as an FP32 pair: differences of the heads round in proportion to themselves, and the
    // remainders restore what the heads lost
    const float g_hi = static_cast<float>(big_g);
    const float g_lo = static_cast<float>(big_g - static_cast<double>(g_hi));
    // this lane's rows g + 8 i and columns 8 i + 2 t (+ 1)
    float rh[4], rl[4], rb[4], ch[8], cl[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      rh[i] = __shfl_sync(0xffffffffu, g_hi, g + 8 * i);
      rl[i] = __shfl_sync(0xffffffffu, g_lo, g + 8 * i);
      rb[i] = __shfl_sync(0xffffffffu, beta, g + 8 * i);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        ch[2 * i + e] = __shfl_sync(0xffffffffu, g_hi, 8 * i + 2 * t + e);
        cl[2 * i + e] = __shfl_sync(0xffffffffu, g_lo, 8 * i + 2 * t + e);
      }
    }
    // rows of X (k or q) times rows of k, the blocks on and below the diagonal:
    // acc[0..1] rows 0..15 x columns 0..15, acc[2..5] rows 16..31 x columns 0..31
    const __half(*xs)[136] = helper == 0 ? sm.k[st] : sm.q[st];
    float acc[6][4];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < D / 16; ++s) {
      uint32_t x0[4], x1[4], k0[4], k1[4];
      const int r = (mat & 1) * 8 + mrow, col = s * 16 + (mat >> 1) * 8;
      ldsm_x4(k0, &sm.k[st][r][col]);
      ldsm_x4(k1, &sm.k[st][16 + r][col]);
      if (helper == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x0[i] = k0[i];
          x1[i] = k1[i];
        }
      } else {
        ldsm_x4(x0, &xs[r][col]);
        ldsm_x4(x1, &xs[16 + r][col]);
      }
      float d[6][4] = {};
      mma16816(d[0], x0[0], x0[1], x0[2], x0[3], k0[0], k0[2]);
      mma16816(d[1], x0[0], x0[1], x0[2], x0[3], k0[1], k0[3]);
      mma16816(d[2], x1[0], x1[1], x1[2], x1[3], k0[0], k0[2]);
      mma16816(d[3], x1[0], x1[1], x1[2], x1[3], k0[1], k0[3]);
      mma16816(d[4], x1[0], x1[1], x1[2], x1[3], k1[0], k1[2]);
      mma16816(d[5], x1[0], x1[1], x1[2], x1[3], k1[1], k1[3]);
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] += d[i][e];
    }
    // every factor first, then the stores: nothing in between waits for shared memory
#pragma unroll
    for (int i = 0; i < 6; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int rn = (i < 2 ? 0 : 2) + (e >> 1), cn = (i < 2 ? i : i - 2) * 2 + (e & 1);
        const float d = (rh[rn] - ch[cn]) + (rl[rn] - cl[cn]);
        acc[i][e] *= expf(fminf(d, 0.f)) * (helper == 0 ? rb[rn] : scale);
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int i0 = i < 2 ? 0 : 16, j0 = i < 2 ? i * 8 : (i - 2) * 8;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ri = i0 + g + (e >> 1) * 8, cj = j0 + 2 * t + (e & 1);
        if (helper == 0) {
          sm.at[cj][ri] = cj < ri ? acc[i][e] : 0.f;
        } else {
          sm.p[buf][ri][cj] = cj < ri ? acc[i][e] : 0.f;
          if (cj == ri) sm.pd[buf][ri] = acc[i][e];
        }
      }
    }
    if (helper == 0) {
      __syncwarp();
      // column `lane` of T by forward substitution: subtract A's column j times T's row j
      float x[CHUNK];
#pragma unroll
      for (int i = 0; i < CHUNK; ++i) x[i] = i == lane ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < CHUNK - 1; ++j) {
#pragma unroll
        for (int i4 = (j + 1) / 4; i4 < CHUNK / 4; ++i4) {
          const float4 a = *reinterpret_cast<const float4*>(&sm.at[j][i4 * 4]);
          if (i4 * 4 > j) x[i4 * 4] = fmaf(-a.x, x[j], x[i4 * 4]);
          if (i4 * 4 + 1 > j) x[i4 * 4 + 1] = fmaf(-a.y, x[j], x[i4 * 4 + 1]);
          if (i4 * 4 + 2 > j) x[i4 * 4 + 2] = fmaf(-a.z, x[j], x[i4 * 4 + 2]);
          x[i4 * 4 + 3] = fmaf(-a.w, x[j], x[i4 * 4 + 3]);
        }
      }
#pragma unroll
      for (int i = 0; i < CHUNK; ++i) sm.t[buf][i][lane] = x[i];
      sm.t[buf][lane][lane] = 0.f;
      __syncwarp();                            // A is rewritten by the next chunk
    }
  };

  if (warp >= 4) {
    stage(0);
    if (chunks > 1) stage(1);
    fetch_gates(0);
  }

  // ---- this warp's slice of S^T: rows dv, columns dk = 8 u + 2 t (+ 1)
  const bool fresh = row_pos[seg.row_start] == 0;
  const int dv = dv0 + (warp & 3) * 16 + g;
  float* sp = state + (static_cast<size_t>(row_slot[seg.row_start]) * hv + vh) * D * D + dv;
  float s_acc[16][4];
  float s_max[2] = {0.f, 0.f};                 // rows g and g + 8
  if (warp < 4) {
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s_acc[u][e] = fresh ? 0.f : sp[(8 * u + 2 * t + (e & 1)) * D + (e >> 1) * 8];
      }
    // a loop of its own: maxima between the loads take them one by one (16 runs of 64 rows: 110 us)
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e) s_max[e >> 1] = fmaxf(s_max[e >> 1], fabsf(s_acc[u][e]));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (warp >= 4) prepare(0);
  __syncthreads();

  for (int c = 0; c < chunks; ++c) {
    if (warp >= 4) {
      if (c + 2 < chunks) stage(c + 2);        // its buffer was last read in round c - 1
      if (c + 1 < chunks) prepare(c + 1);
    } else {
      const int st = c % 3, buf = c & 1;
      float up[2], down[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = bound_exp(quad_max(s_max[h]));
        up[h] = pow2i(14 - e);
        down[h] = pow2i(e - 14);
      }
      // ---- S^T k and S^T q: columns are the chunk's rows
      float ak[4][4], aq[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ak[i][j] = aq[i][j] = 0.f;
#pragma unroll
      for (int s = 0; s < D / 16; s += 2) {
        uint32_t hi[2][4], lo[2][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float* x = s_acc[2 * s + (i >> 1)] + (i & 1) * 2;
          split_half2(x[0] * up[i & 1], x[1] * up[i & 1], hi[i >> 2][i & 3], lo[i >> 2][i & 3]);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int x = 0; x < 2; ++x) {              // k, then q
            uint32_t b[2][4];
            const int r = half * 16 + (mat >> 1) * 8 + mrow, col = s * 16 + (mat & 1) * 8;
            ldsm_x4(b[0], &(x == 0 ? sm.k : sm.q)[st][r][col]);
            ldsm_x4(b[1], &(x == 0 ? sm.k : sm.q)[st][r][col + 16]);
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              float part[4] = {};
              mma16816(part, lo[0][0], lo[0][1], lo[0][2], lo[0][3], b[0][2 * v], b[0][2 * v + 1]);
              mma16816(part, lo[1][0], lo[1][1], lo[1][2], lo[1][3], b[1][2 * v], b[1][2 * v + 1]);
              mma16816(part, hi[0][0], hi[0][1], hi[0][2], hi[0][3], b[0][2 * v], b[0][2 * v + 1]);
              mma16816(part, hi[1][0], hi[1][1], hi[1][2], hi[1][3], b[1][2 * v], b[1][2 * v + 1]);
              float(&to)[4] = (x == 0 ? ak : aq)[half * 2 + v];
#pragma unroll
              for (int e = 0; e < 4; ++e) to[e] += part[e];
            }
          }
      }
      // ---- B^T, and e^G S^T q as the start of the output
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int r = 8 * v + 2 * t;
        const float2 eg = *reinterpret_cast<const float2*>(&sm.eg[buf][r]);
        const float2 be = *reinterpret_cast<const float2*>(&sm.beta[buf][r]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float ge = (e & 1 ? eg.y : eg.x) * down[e >> 1];
          const float val = __half2float(sm.v[st][r + (e & 1)][(warp & 3) * 16 + g + (e >> 1) * 8]);
          ak[v][e] = (e & 1 ? be.y : be.x) * fmaf(-ge, ak[v][e], val);
          aq[v][e] *= ge * scale;
        }
      }
      // the diagonals carry most of both sums: they are multiplied in FP32
      float dl[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dl[i][j] = ak[i][j];
      mul_lower(dl, ak, sm.t[buf], g, t);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float2 pd = *reinterpret_cast<const float2*>(&sm.pd[buf][8 * v + 2 * t]);
#pragma unroll
        for (int e = 0; e < 4; ++e) aq[v][e] = fmaf(e & 1 ? pd.y : pd.x, dl[v][e], aq[v][e]);
      }
      mul_lower(aq, dl, sm.p[buf], g, t);
      const int n = min(CHUNK, seg.rows - c * CHUNK);
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = 8 * v + 2 * t + (e & 1);
          if (r < n)
            out[(static_cast<size_t>(seg.row_start + c * CHUNK + r) * hv + vh) * D + dv +
                (e >> 1) * 8] = aq[v][e];
        }
      // ---- state update
      float d_max[2] = {0.f, 0.f};
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const float2 tl = *reinterpret_cast<const float2*>(&sm.tail[buf][8 * v + 2 * t]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          dl[v][e] *= e & 1 ? tl.y : tl.x;
          d_max[e >> 1] = fmaxf(d_max[e >> 1], fabsf(dl[v][e]));
        }
      }
      float dup[2], ddown[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = bound_exp(quad_max(d_max[h]));
        dup[h] = pow2i(14 - e);
        ddown[h] = pow2i(e - 14);
      }
      const float total = sm.total[buf];
      s_max[0] = s_max[1] = 0.f;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        // head, remainder and its remainder: a new row of S is this product to the last bit
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          split_half3(dl[2 * r + (i >> 1)][(i & 1) * 2] * dup[i & 1],
                      dl[2 * r + (i >> 1)][(i & 1) * 2 + 1] * dup[i & 1], hi[i], mid[i], lo[i]);
#pragma unroll
        for (int u = 0; u < 16; u += 2) {
          uint32_t b[4];
          float add[2][4] = {};
          ldsm_x4_t(b, &sm.k[st][r * 16 + (mat & 1) * 8 + mrow][(u + (mat >> 1)) * 8]);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            mma16816(add[j], lo[0], lo[1], lo[2], lo[3], b[2 * j], b[2 * j + 1]);
            mma16816(add[j], mid[0], mid[1], mid[2], mid[3], b[2 * j], b[2 * j + 1]);
            mma16816(add[j], hi[0], hi[1], hi[2], hi[3], b[2 * j], b[2 * j + 1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float& x = s_acc[u + j][e];
              x = r == 0 ? fmaf(x, total, add[j][e] * ddown[e >> 1])
                         : fmaf(add[j][e], ddown[e >> 1], x);
              if (r == 1) s_max[e >> 1] = fmaxf(s_max[e >> 1], fabsf(x));
            }
          }
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  if (warp < 4) {
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        sp[(8 * u + 2 * t + (e & 1)) * D + (e >> 1) * 8] = s_acc[u][e];
  }
}

// Replays the first accepted[seg] recorded steps of every segment onto the stored state:
// S = decay * S + k (x) delta, in row order.  Same thread layout as the scan.
template <int D>
__global__ void __launch_bounds__(256) gdn_commit_kernel(
    const float* __restrict__ factors, const Segment* __restrict__ segs,
    const int* __restrict__ accepted, const int* __restrict__ row_slot,
    const int* __restrict__ row_pos, int hv, float* __restrict__ state) {
  constexpr int PARTS = 256 / D, ROWS = D / PARTS;
  const int vh = blockIdx.x;
  const Segment seg = segs[blockIdx.y];
  const int steps = min(accepted[blockIdx.y], seg.rows);
  if (steps <= 0) return;
  const int dv = threadIdx.x % D, part_id = threadIdx.x / D;
  const int slot = row_slot[seg.row_start];
  const bool fresh = row_pos[seg.row_start] == 0;
  float* sp = state + ((static_cast<size_t>(slot) * hv + vh) * D + part_id * ROWS) * D + dv;
  float s[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) s[i] = fresh ? 0.f : sp[static_cast<size_t>(i) * D];
  for (int t = 0; t < steps; ++t) {
    const float* f =
        factors + (static_cast<size_t>(seg.row_start + t) * hv + vh) * (2 * D + 1);
    const float decay = f[0], delta = f[1 + D + dv];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) s[i] = fmaf(f[1 + part_id * ROWS + i], delta, s[i] * decay);
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) sp[static_cast<size_t>(i) * D] = s[i];
}

// ---------------------------------------------------------------- gated norm
// grid (rows, HV), D threads: y = rmsnorm(o) * w * silu(z)  (sigmoid(z) when sigmoid_gate).  The
// sum of squares is built as in the warp form below, so a row gives the same bits through both.
template <int D>
__global__ void __launch_bounds__(D) gdn_gated_norm_kernel(
    const float* o, const __half* z, int z_stride, const __half* w, float eps, int sigmoid_gate,
    int hv, __half* __restrict__ y) {
  grid_wait();
  grid_release();
  const int row = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
  const float v = o[(static_cast<size_t>(row) * hv + h) * D + d];
  constexpr int V = D / 32;
  __shared__ float red[32];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const float x = __shfl_sync(0xffffffffu, v, (d & 31 & ~(V - 1)) + i);
    ss = fmaf(x, x, ss);
  }
  if (d % V == 0) red[d / V] = ss;
  __syncthreads();
  const float tot = warp_sum(red[d & 31]);
  const float n = v * rsqrtf(tot / D + eps) * __half2float(w[d]);
  const float zf = __half2float(z[static_cast<size_t>(row) * z_stride + h * D + d]);
  const float sg = sigmoid_pair(make_float2(zf, zf)).x;       // the bits of the form below
  const float gate = sigmoid_gate ? sg : zf * sg;
  y[(static_cast<size_t>(row) * hv + h) * D + d] = __float2half_rn(n * gate);
}

// The same, one warp per (row, head): D / 32 neighbouring channels per lane, no block barrier.
// 2600 rows x 32 heads of 128: 45 -> 19 us (85 MB); 2100 rows 17 -> 15 with two values to an
// instruction (68 MB).  A few heads are quicker with a thread per
// channel, which computes one sigmoid instead of four: 4 rows x 32 heads 1.2 us against 1.6, 48
// rows 1.9 against 2.0, 64 rows 2.1 against 2.0.
template <int D>
__global__ void __launch_bounds__(256) gdn_gated_norm_warp_kernel(
    const float* o, const __half* z, int z_stride, const __half* w, float eps, int sigmoid_gate,
    int hv, long long items, __half* __restrict__ y) {
  constexpr int V = D / 32;
  struct __align__(V * 2) Half {
    __half h[V];
  };
  struct __align__(V * 4) Float {
    float f[V];
  };
  grid_wait();
  grid_release();
  const long long item = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (item >= items) return;
  const int lane = threadIdx.x & 31;
  const long long row = item / hv;
  const int h = static_cast<int>(item - row * hv);
  const Float v = *reinterpret_cast<const Float*>(o + item * D + lane * V);
  const Half zh = *reinterpret_cast<const Half*>(z + row * z_stride + h * D + lane * V);
  const Half wh = *reinterpret_cast<const Half*>(w + lane * V);
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) ss = fmaf(v.f[i], v.f[i], ss);
  const float r = rsqrtf(warp_sum(ss) / D + eps);
  Half out;
#pragma unroll
  for (int i = 0; i < V; i += 2) {
    const float2 zf = make_float2(__half2float(zh.h[i]), __half2float(zh.h[i + 1]));
    const float2 wf = make_float2(__half2float(wh.h[i]), __half2float(wh.h[i + 1]));
    const float2 n = mul2(mul2(make_float2(v.f[i], v.f[i + 1]), make_float2(r, r)), wf);
    const float2 sg = sigmoid_pair(zf);
    const float2 res = mul2(n, sigmoid_gate ? sg : mul2(zf, sg));
    out.h[i] = __float2half_rn(res.x);
    out.h[i + 1] = __float2half_rn(res.y);
  }
  *reinterpret_cast<Half*>(y + item * D + lane * V) = out;
}

inline bool aligned(const void* p, size_t bytes) {
  return reinterpret_cast<uintptr_t>(p) % bytes == 0;
}

template <int D>
static void launch_conv(const __half* x, int x_stride, const __half* weight, const __half* hist,
                        const int* row_first, const int* row_slot, const int* row_pos, int rows,
                        int conv_dim, int hk, __half* y, cudaStream_t stream) {
  const bool vec = x_stride % 8 == 0 && aligned(x, 16) && aligned(weight, 16) &&
                   aligned(hist, 16) && aligned(y, 16);
  if (!vec) {
    gdn_conv_kernel<D><<<dim3(rows, conv_dim / D), D, 0, stream>>>(
        x, x_stride, weight, hist, row_first, row_slot, row_pos, conv_dim, 2 * hk, y);
    return;
  }
  const int cols = (conv_dim + 2047) / 2048;
  const int most = 2 * 148 / cols > 1 ? 2 * 148 / cols : 1;      // strips at once
  const int strip = (rows + most - 1) / most;
  const dim3 grid((rows + strip - 1) / strip, cols);
  auto kernel = strip > 1 ? gdn_conv_vec_kernel<D, 4> : gdn_conv_vec_kernel<D, 1>;
  launch_early(kernel, grid, 256, 0, stream, x, x_stride, weight, hist, row_first, row_slot,
               row_pos, rows, conv_dim, 2 * hk * D, strip, y);
}

static void launch_history(const __half* x, int x_stride, const Segment* segs, int n_segs,
                           const int* row_slot, const int* row_pos, int conv_dim, __half* hist,
                           const int* accepted, cudaStream_t stream) {
  if (x_stride % 8 == 0 && aligned(x, 16) && aligned(hist, 16))
    launch_early(gdn_history_kernel<8>, dim3(n_segs, (conv_dim + 2047) / 2048), 256, 0, stream, x,
                 x_stride, segs, row_slot, row_pos, conv_dim, hist, accepted);
  else
    launch_early(gdn_history_kernel<1>, dim3(n_segs, (conv_dim + 255) / 256), 256, 0, stream, x,
                 x_stride, segs, row_slot, row_pos, conv_dim, hist, accepted);
}

// Whether long runs take the kernel of gdn_pipe.cu: where its CTAs have an SM each, or the runs are
// long enough to make up for their waves (figures there).  A caller that does not know the longest
// run gives the rows in all.
static bool gdn_pipelined(int hv, int n_segs, int max_seg_rows) {
  return 2LL * hv * n_segs <= 148 || max_seg_rows >= 384LL * n_segs;
}

}  // namespace orinfer

using namespace orinfer;

extern "C" {

int orinfer_gdn_pipelined(int hv, int n_segs, int max_seg_rows) {
  return gdn_pipelined(hv, n_segs, max_seg_rows) ? 1 : 0;
}

int orinfer_small_proj(const __half* x, const __half* w, float* out, int rows, int hidden, int n,
                       cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (hidden % 8) return -1;
  launch_early(small_proj_kernel, rows, 256, 0, stream, x, w, out, hidden, n);
  return static_cast<int>(cudaGetLastError());
}

// x: fp16 [rows, x_stride] with q|k|v in the first conv_dim channels; y: fp16 [rows, conv_dim].
// segs: int32 [n_segs, 4] = (first row, rows, 0, 0).  Updates hist in place.
int orinfer_gdn_conv(const __half* x, int x_stride, const __half* weight, __half* hist,
                     const int* row_first, const int* row_slot, const int* row_pos,
                     const int* segs, int n_segs,
                     int rows, int hk, int hv, int head_dim, __half* y, cudaStream_t stream,
                     int update_history) {
  if (rows <= 0) return 0;
  if (head_dim != 128 && head_dim != 64) return -1;
  const int conv_dim = (2 * hk + hv) * head_dim;
  if (head_dim == 128)
    launch_conv<128>(x, x_stride, weight, hist, row_first, row_slot, row_pos, rows, conv_dim, hk, y,
                     stream);
  else
    launch_conv<64>(x, x_stride, weight, hist, row_first, row_slot, row_pos, rows, conv_dim, hk, y,
                    stream);
  if (update_history && n_segs > 0)
    launch_history(x, x_stride, reinterpret_cast<const Segment*>(segs), n_segs, row_slot, row_pos,
                   conv_dim, hist, nullptr, stream);
  return static_cast<int>(cudaGetLastError());
}

// Commit of a verification pass: advances the convolution history by the first accepted[s]
// rows of every segment (x = the pre-convolution rows kept from the pass) and replays the
// recorded state updates of those rows.
int orinfer_gdn_commit(const __half* x, int x_stride, const float* factors, const int* segs,
                       int n_segs, const int* accepted, const int* row_slot, const int* row_pos,
                       int hk, int hv, int head_dim, __half* hist, float* state,
                       cudaStream_t stream) {
  if (n_segs <= 0) return 0;
  if (head_dim != 128 && head_dim != 64) return -1;
  const Segment* sg = reinterpret_cast<const Segment*>(segs);
  const int conv_dim = (2 * hk + hv) * head_dim;
  launch_history(x, x_stride, sg, n_segs, row_slot, row_pos, conv_dim, hist, accepted, stream);
  if (head_dim == 128)
    gdn_commit_kernel<128><<<dim3(hv, n_segs), 256, 0, stream>>>(factors, sg, accepted, row_slot,
                                                                row_pos, hv, state);
  else
    gdn_commit_kernel<64><<<dim3(hv, n_segs), 256, 0, stream>>>(factors, sg, accepted, row_slot,
                                                               row_pos, hv, state);
  return static_cast<int>(cudaGetLastError());
}

// qkv: conv output fp16 [rows, conv_dim]; ab fp32 [rows, 2*HV]; state fp32 (below);
// out fp32 [rows, HV, D].  head_dim D is 64 or 128; state is [slots, HV, D, D].
int orinfer_gdn_scan(const __half* qkv, const float* ab, const float* a_log, const float* dt_bias,
                     const int* segs, int n_segs, const int* row_slot, const int* row_pos, int hk,
                     int hv, int head_dim, float* state, float* out, cudaStream_t stream,
                     float* factors, int max_seg_rows) {
  if (n_segs <= 0) return 0;
  if ((head_dim != 128 && head_dim != 64) || hv % hk) return -1;
  const Segment* sg = reinterpret_cast<const Segment*>(segs);
  const int conv_dim = (2 * hk + hv) * head_dim;
  // Few CTAs at one per head (prefill of a few long segments, small decode batches): spread
  // each head over D/32 CTAs.  The rule depends on the segment count only, so a verification
  // pass and the plain pass over the same requests take the same arithmetic.
  const bool split = static_cast<long long>(hv) * n_segs < 2 * 148;
  // Runs of at least GDN_LONG_ROWS rows take the chunked kernel (which skips the others, as the
  // scan skips them); verification passes and 64-channel heads never do.  Which runs are long only
  // the device knows, and a launch that finds none costs 1.5 to 3 us (8 runs of 20 rows: 48 -> 51
  // us), so a packet of several runs that leaves one at most 63 rows does without: one run among
  // them of 40 to 63 rows loses up to 9 us by that.
  int long_rows = 0x7fffffff;
  if (head_dim == 128 && factors == nullptr && aligned(qkv, 16) &&
      max_seg_rows >= (n_segs == 1 ? GDN_LONG_ROWS : 64)) {
    long_rows = GDN_LONG_ROWS;
    // (it moves state and outputs in pairs)
    if (gdn_pipelined(hv, n_segs, max_seg_rows) && aligned(state, 8) && aligned(out, 8)) {
      if (const int e = gdn_pipe_launch(qkv, conv_dim, ab, a_log, dt_bias, sg, n_segs, row_slot,
                                        row_pos, hk, hv, state, out, stream))
        return e;
    } else {
      static const int slot = runtime_new_slot();
      if (const int e = runtime_allow_smem(slot, gdn_chunk_kernel, sizeof(ChunkSmem))) return e;
      // Not early: its few long CTAs would gather, two to an SM, where the kernel before ends
      // first (the mixer of two runs of 1050 rows 260 us, 245 so, of two of 1500 357 and 335).
      gdn_chunk_kernel<<<dim3(hv * 2, n_segs), CHUNK_THREADS, sizeof(ChunkSmem), stream>>>(
          qkv, conv_dim, ab, a_log, dt_bias, sg, row_slot, row_pos, hk, hv, state, out);
    }
  }
#define ORINFER_SCAN(KERNEL, GRID_X)                                                       \
  launch_early(KERNEL, dim3(GRID_X, n_segs), 256, 0, stream, qkv, conv_dim, ab, a_log,     \
               dt_bias, sg, row_slot, row_pos, hk, hv, state, out, factors, long_rows)
  if (head_dim == 128) {
    if (split) ORINFER_SCAN(gdn_scan_split_kernel<128>, hv * 4);
    else ORINFER_SCAN((gdn_scan_kernel<128, 128>), hv);
  } else {
    if (split) ORINFER_SCAN(gdn_scan_split_kernel<64>, hv * 2);
    else ORINFER_SCAN((gdn_scan_kernel<64, 64>), hv);
  }
#undef ORINFER_SCAN
  return static_cast<int>(cudaGetLastError());
}

int orinfer_gdn_gated_norm(const float* o, const __half* z, int z_stride, const __half* w,
                           float eps, int sigmoid_gate, int rows, int hv, int head_dim,
                           __half* y, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (head_dim != 128 && head_dim != 64) return -1;
  const int v = head_dim / 32;
  const long long items = static_cast<long long>(rows) * hv;
  if (items >= 1536 && z_stride % v == 0 && aligned(z, 2 * v) && aligned(w, 2 * v) &&
      aligned(o, 4 * v) && aligned(y, 2 * v)) {
    const unsigned grid = static_cast<unsigned>((items + 7) / 8);
    if (head_dim == 128)
      launch_early(gdn_gated_norm_warp_kernel<128>, grid, 256, 0, stream, o, z, z_stride, w, eps,
                                                               sigmoid_gate, hv, items, y);
    else
      launch_early(gdn_gated_norm_warp_kernel<64>, grid, 256, 0, stream, o, z, z_stride, w, eps,
                                                              sigmoid_gate, hv, items, y);
    return static_cast<int>(cudaGetLastError());
  }
  if (head_dim == 128)
    launch_early(gdn_gated_norm_kernel<128>, dim3(rows, hv), 128, 0, stream, o, z, z_stride, w, eps,
                                                                   sigmoid_gate, hv, y);
  else if (head_dim == 64)
    launch_early(gdn_gated_norm_kernel<64>, dim3(rows, hv), 64, 0, stream, o, z, z_stride, w, eps,
                                                                 sigmoid_gate, hv, y);
  else
    return -1;
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
