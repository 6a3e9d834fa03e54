// Reductions (sum, mean, max, min) with the reference's summation tree, one read of the
// input instead of the reference's transpose + log2(COLS) in-place stages + slice
// (litenn/core/op/reduce.py:166-205, stage kernel :279-293).
//
// The reference reduces a row of n values in stages: h = ceil(n/2); x[c] = x[c] (+) x[c+h]
// for every c with c+h < n; n = h; until n == 1.  With n_0 = COLS and n_j = ceil(n_{j-1}/2)
// the value at stage s, column c is V_s(c) = V_{s-1}(c) (+) V_{s-1}(c + n_s) when that
// partner exists, else V_{s-1}(c).  Here one thread evaluates a whole subtree V_s(c0), so
// the operand pairing, and therefore every rounding, is the reference's.  The leaves of
// V_s(c0) are c0 plus any subset of {n_1 .. n_s}, minus the subsets that step over the end of
// a stage of odd length; neighbouring c0 read neighbouring leaves, so every load is coalesced.
// A row is finished inside a warp (shuffles), inside a block (shared memory), or, when a
// row is split over many threads to fill the GPU, by running the same routine again on the
// partial values -- the tree over n_s partials is the tail of the tree over n_0 values.
#include "lnn_common.cuh"
#include <math_constants.h>
#include <utility>
#include <algorithm>

using lnn::FastDiv;

namespace {

constexpr int kThreads = 256;
constexpr int kMaxLevels = 40;
constexpr int kMaxPow2Levels = 9;      // leaves per thread of a split row: at most 2^9

struct Levels {
  int S;                       // number of stages: n[S] == 1
  int pow2;                    // COLS is a power of two
  int exact;                   // number of leading stages that halve an even length
  uint32_t n[kMaxLevels + 1];  // n[0] = COLS, n[j] = ceil(n[j-1]/2)
};

struct RedGeom {
  int64_t outer, r0, mid, r1, inner;
  int64_t rows;        // outer*mid*inner
  int64_t stride_r0;   // mid*r1*inner
  int64_t stride_r1;   // inner
  int64_t stride_outer;// r0*mid*r1*inner
  int64_t stride_mid;  // r1*inner
  int small;           // every element index fits 31 bits
  FastDiv by_r0, by_mid, by_r1, by_inner;
};

template <int OP>
__device__ __forceinline__ float comb(float a, float b) {
  if (OP == LNN_RED_MAX) return fmaxf(a, b);
  if (OP == LNN_RED_MIN) return fminf(a, b);
  return __fadd_rn(a, b);
}
template <int OP>
__device__ __forceinline__ float4 comb(const float4& a, const float4& b) {
  return make_float4(comb<OP>(a.x, b.x), comb<OP>(a.y, b.y), comb<OP>(a.z, b.z), comb<OP>(a.w, b.w));
}
__device__ __forceinline__ void load_leaf(float& v, const float* p) { v = __ldcs(p); }
__device__ __forceinline__ void load_leaf(float4& v, const float* p) { v = __ldcs(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void set_zero(float& v) { v = 0.0f; }
__device__ __forceinline__ void set_zero(float4& v) { v = make_float4(0.f, 0.f, 0.f, 0.f); }

// What a finished row stores: O (+)= v / COLS (mean) or v.
__device__ __forceinline__ void finish(float* O, float v, int acc, float mean_div) {
  if (mean_div != 0.0f) v = __fdiv_rn(v, mean_div);
  *O = acc ? __fadd_rn(*O, v) : v;
}
__device__ __forceinline__ void finish(float* O, float4 v, int acc, float mean_div) {
  if (mean_div != 0.0f) {
    v.x = __fdiv_rn(v.x, mean_div); v.y = __fdiv_rn(v.y, mean_div);
    v.z = __fdiv_rn(v.z, mean_div); v.w = __fdiv_rn(v.w, mean_div);
  }
  float4* dst = reinterpret_cast<float4*>(O);
  if (acc) v = comb<LNN_RED_SUM>(*dst, v);
  *dst = v;
}

__device__ __forceinline__ int64_t row_base(const RedGeom& g, int64_t row) {
  if (g.small) {
    const uint32_t t = g.by_inner.div((uint32_t)row);
    const uint32_t outer_i = g.by_mid.div(t);
    return (int64_t)outer_i * g.stride_outer + (int64_t)(t - outer_i * g.by_mid.d) * g.stride_mid +
           ((uint32_t)row - t * g.by_inner.d);
  }
  const int64_t inner_i = row % g.inner;
  const int64_t t = row / g.inner;
  const int64_t mid_i = t % g.mid;
  const int64_t outer_i = t / g.mid;
  return outer_i * g.stride_outer + mid_i * g.stride_mid + inner_i;
}

__device__ __forceinline__ int64_t leaf_offset(const RedGeom& g, uint32_t leaf) {
  if (g.r0 == 1) return (int64_t)leaf * g.stride_r1;
  const uint32_t q = g.by_r1.div(leaf);
  return (int64_t)q * g.stride_r0 + (int64_t)(leaf - q * g.by_r1.d) * g.stride_r1;
}

// V_s(c0) of one row (base points at the row's column 0); V = float, or float4 for four adjacent
// kept rows or four adjacent columns at once.  The leaves of the first LA stages are loaded together
// (2^LA independent loads in flight) and paired in registers, stage 1 first; the later stages run
// over t, whose bit k takes the partner of stage LA + 1 + k, with one waiting value per stage (a
// binary counter: t counts up, so a left operand is always complete before its right one).
// EXACT: every stage up to s halves an even length (and s >= LA), so no partner is ever missing.
template <int OP, class V, int LA, bool EXACT>
__device__ __forceinline__ V subtree_of(const float* __restrict__ base, uint32_t c0, int s, const Levels& L,
                                        const RedGeom& g) {
  constexpr int A = 1 << LA;
  const int lb = s > LA ? s - LA : 0;
  V stack[kMaxLevels - LA];
  uint32_t waiting = 0;                          // which entries of stack hold a value that exists
  V w;
  set_zero(w);
  for (uint32_t t = 0; t < (1u << lb); ++t) {
    uint32_t cur = c0;
    bool have = true;
    for (int k = lb - 1; k >= 0; --k)
      if ((t >> k) & 1u) {
        cur += L.n[LA + 1 + k];
        if (!EXACT) have = have && cur < L.n[LA + k];
      }
    if (EXACT || have) {
      V v[A];
      if (EXACT) {
#pragma unroll
        for (int a = 0; a < A; ++a) load_leaf(v[a], base + leaf_offset(g, cur + (uint32_t)a * L.n[LA]));
#pragma unroll
        for (int h = A / 2; h >= 1; h >>= 1)
#pragma unroll
          for (int i = 0; i < h; ++i) v[i] = comb<OP>(v[i], v[i + h]);
      } else {
        uint32_t id[A];
        bool ok[A];
        id[0] = cur; ok[0] = true;
#pragma unroll
        for (int j = LA; j >= 1; --j)              // bit LA - j of the leaf number takes stage j's partner
#pragma unroll
          for (int a = 0; a < (1 << (LA - j)); ++a) {
            const int b = a | (1 << (LA - j));
            id[b] = id[a] + L.n[j];
            ok[b] = ok[a] && j <= s && id[b] < L.n[j - 1];
          }
#pragma unroll
        for (int a = 0; a < A; ++a) {
          set_zero(v[a]);
          if (ok[a]) load_leaf(v[a], base + leaf_offset(g, id[a]));
        }
#pragma unroll
        for (int h = A / 2; h >= 1; h >>= 1)
#pragma unroll
          for (int i = 0; i < h; ++i)
            if (ok[i + h]) v[i] = comb<OP>(v[i], v[i + h]);
      }
      w = v[0];
    }
    int level = 0;
    for (uint32_t tt = t; tt & 1u; tt >>= 1, ++level) {
      if (EXACT) { w = comb<OP>(stack[level], w); continue; }
      if (have) w = comb<OP>(stack[level], w);     // a left operand is never missing when its partner exists
      else { w = stack[level]; have = (waiting >> level) & 1u; }
    }
    stack[level] = w;
    waiting = (waiting & ~(1u << level)) | ((uint32_t)have << level);
  }
  return w;
}

// V_S(c0) for S stages known at compile time: one batch of 2^S loads and no loop.
template <int OP, class V, int S>
__device__ __forceinline__ V subtree_of_stages(const float* __restrict__ base, uint32_t c0, const Levels& L, const RedGeom& g) {
  if (S <= L.exact) return subtree_of<OP, V, S, true>(base, c0, S, L, g);
  return subtree_of<OP, V, S, false>(base, c0, S, L, g);
}
template <class V> struct LoadStages { static constexpr int value = 4; };      // 16 scalar loads in flight
template <> struct LoadStages<float4> { static constexpr int value = 3; };     // 8 vector loads
template <int OP, class V>
__device__ __forceinline__ V subtree(const float* __restrict__ base, uint32_t c0, int s, const Levels& L,
                                     const RedGeom& g) {
  constexpr int LA = LoadStages<V>::value;
  if (s >= LA && s <= L.exact) return subtree_of<OP, V, LA, true>(base, c0, s, L, g);
  return subtree_of<OP, V, LA, false>(base, c0, s, L, g);
}

// Short rows.  W consecutive lanes share a row (32 / W rows per warp): lane t owns subtree c0 = t of the n[S] <= W
// that are left after S stages, one batch of loads, and the last stages are shuffles: lane t takes lane
// t + n_j.  inner == 1: neighbouring lanes read neighbouring columns (W > 1) or rows whose elements share
// sectors (W == 1); inner > 1 (W == 1 only): neighbouring rows.
template <int OP, int W, int S>
__global__ void __launch_bounds__(kThreads)
reduce_rows_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L, int acc, float mean_div) {
  const int lane = threadIdx.x & 31, t = lane & (W - 1);
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row0 = warp0 * (32 / W); row0 < g.rows; row0 += nwarps * (32 / W)) {
    const int64_t row = row0 + lane / W;
    float v = 0.0f;
    if (row < g.rows && t < (int)L.n[S]) v = subtree_of_stages<OP, float, S>(I + row_base(g, row), (uint32_t)t, L, g);
    if (W > 1)
      for (int j = S + 1; j <= L.S; ++j) {
        const int h = (int)L.n[j];
        const float other = __shfl_down_sync(0xffffffffu, v, h, W);
        if (t + h < (int)L.n[j - 1]) v = comb<OP>(v, other);
      }
    if (t == 0 && row < g.rows) finish(O + row, v, acc, mean_div);
  }
}

// inner == 1, n[s] <= 32: one warp per row.  Lane t owns subtree c0 = t (coalesced: neighbouring
// lanes read neighbouring columns) and the last stages are shuffles: lane t takes lane t + n_j.
template <int OP>
__global__ void __launch_bounds__(kThreads)
reduce_warp_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L, int s,
                   int acc, float mean_div) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp0; row < g.rows; row += nwarps) {
    float v = 0.0f;
    if (lane < (int)L.n[s]) v = subtree<OP, float>(I + row_base(g, row), (uint32_t)lane, s, L, g);
    for (int j = s + 1; j <= L.S; ++j) {
      const int h = (int)L.n[j];
      const float other = __shfl_down_sync(0xffffffffu, v, h);
      if (lane + h < (int)L.n[j - 1]) v = comb<OP>(v, other);
    }
    if (lane == 0) finish(O + row, v, acc, mean_div);
  }
}

// inner == 1, n[s] <= tpr <= 256: tpr consecutive threads share a row, thread t owns subtree
// c0 = t, and the remaining stages s+1..S run in shared memory.
template <int OP>
__global__ void __launch_bounds__(kThreads)
reduce_rowcoop_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L,
                      int s, int tpr, int acc, float mean_div) {
  __shared__ float vals[kThreads];
  const int rows_per_block = kThreads / tpr;
  const int t = threadIdx.x & (tpr - 1);
  const int64_t row = (int64_t)blockIdx.x * rows_per_block + threadIdx.x / tpr;
  const bool active = row < g.rows && t < (int)L.n[s];
  float v = 0.0f;
  if (active) v = subtree<OP, float>(I + row_base(g, row), (uint32_t)t, s, L, g);
  vals[threadIdx.x] = v;
  __syncthreads();
  for (int j = s + 1; j <= L.S; ++j) {
    const int nj = (int)L.n[j];
    const bool doit = active && t + nj < (int)L.n[j - 1];
    if (doit) v = comb<OP>(v, vals[threadIdx.x + nj]);
    __syncthreads();
    if (doit) vals[threadIdx.x] = v;
    __syncthreads();
  }
  if (active && t == 0) finish(O + row, v, acc, mean_div);
}

// inner > 1: a block takes 32 adjacent kept rows (32 groups of four with V = float4) and splits their
// columns over its eight warps: warp w owns the subtree c0 = w of the n[s] <= 8 that are left, whose
// values meet in shared memory for the remaining stages.  One launch and no partials in memory; 64 leaves per
// thread of [256, 512, 1024] over axis 1 read at 6.2 TB/s, where four partial rows through memory
// and a second launch gave 5.4.
constexpr int kColParts = kThreads / 32;
template <int OP, class V>
__global__ void __launch_bounds__(kThreads)
reduce_cols_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L, int s, int acc,
                   float mean_div) {
  constexpr int VW = sizeof(V) / 4;
  __shared__ V vals[kColParts][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int parts = (int)L.n[s];
  const int64_t groups = g.rows / VW;
  for (int64_t g0 = (int64_t)blockIdx.x * 32; g0 < groups; g0 += (int64_t)gridDim.x * 32) {
    const int64_t row = (g0 + lane) * VW;
    const bool real = g0 + lane < groups;
    const float* base = I + row_base(g, real ? row : 0);
    if (real && warp < parts) {
      // few columns: sixteen predicated loads for the one to eight there are cost more than a branch on s does
      // (scalar loads only: the vector instance needs a third more registers for it)
      if (VW == 1 && s == 0) vals[warp][lane] = subtree_of_stages<OP, V, 0>(base, (uint32_t)warp, L, g);
      else if (VW == 1 && s == 1) vals[warp][lane] = subtree_of_stages<OP, V, 1>(base, (uint32_t)warp, L, g);
      else if (VW == 1 && s == 2) vals[warp][lane] = subtree_of_stages<OP, V, 2>(base, (uint32_t)warp, L, g);
      else if (VW == 1 && s == 3) vals[warp][lane] = subtree_of_stages<OP, V, 3>(base, (uint32_t)warp, L, g);
      else vals[warp][lane] = subtree<OP, V>(base, (uint32_t)warp, s, L, g);
    }
    __syncthreads();
    for (int j = s + 1; j <= L.S; ++j) {
      const int nj = (int)L.n[j];
      if (real && warp + nj < (int)L.n[j - 1]) vals[warp][lane] = comb<OP>(vals[warp][lane], vals[warp + nj][lane]);
      __syncthreads();
    }
    if (warp == 0 && real) finish(O + row, vals[0][lane], acc, mean_div);
    __syncthreads();
  }
}

// One thread per (row, c0) pair evaluating V_s(c0); parts = n[s].  c0_fastest selects which
// index varies between neighbouring threads (columns when the reduced axis is the
// contiguous one, rows when an inner kept axis is).  V = float4: four adjacent columns (c0_fastest) or
// four adjacent kept rows.  parts == 1 finishes rows and writes O; otherwise partials go to P laid
// out [row][parts] (c0_fastest) or [outer][parts][mid*inner].
template <int OP, class V>
__global__ void __launch_bounds__(kThreads, 4)
reduce_parts_kernel(float* __restrict__ O, float* __restrict__ P, const float* __restrict__ I,
                    RedGeom g, Levels L, int s, int c0_fastest, int acc, float mean_div) {
  constexpr int VW = sizeof(V) / 4;
  const int64_t parts = L.n[s];
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const int64_t mi = g.mid * g.inner;
  const int64_t rows = c0_fastest ? g.rows : g.rows / VW, cparts = c0_fastest ? parts / VW : parts;
  const int64_t total = rows * cparts;
  for (int64_t gid = tid; gid < total; gid += nthreads) {
    int64_t c0, row;
    if (c0_fastest) { row = gid / cparts; c0 = (gid - row * cparts) * VW; }
    else { c0 = gid / rows; row = (gid - c0 * rows) * VW; }
    const V v = subtree<OP, V>(I + row_base(g, row), (uint32_t)c0, s, L, g);
    if (parts == 1) {
      finish(O + row, v, acc, mean_div);
    } else if (c0_fastest) {
      *reinterpret_cast<V*>(P + row * parts + c0) = v;      // partials of a row are contiguous
    } else {
      const int64_t outer_i = row / mi;
      *reinterpret_cast<V*>(P + (outer_i * parts + c0) * mi + (row - outer_i * mi)) = v;
    }
  }
}

// inner == 1, power-of-two COLS >= 128, contiguous columns: one warp per row with 128-bit
// loads.  Lane t owns the four subtrees c0 = 4t..4t+3 of the n[s] = 128 partials; the last
// stages pair c with c+64 ... c+4 by shuffles (lane t with t+16 ... t+1), then c with c+2
// and c with c+1 inside the lane.
template <int OP>
__global__ void __launch_bounds__(kThreads)
reduce_warp4_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L, int s,
                    int acc, float mean_div) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp0; row < g.rows; row += nwarps) {
    float4 v = subtree<OP, float4>(I + row_base(g, row), 4u * lane, s, L, g);
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
      float4 o;
      o.x = __shfl_down_sync(0xffffffffu, v.x, h); o.y = __shfl_down_sync(0xffffffffu, v.y, h);
      o.z = __shfl_down_sync(0xffffffffu, v.z, h); o.w = __shfl_down_sync(0xffffffffu, v.w, h);
      if (lane < h) v = comb<OP>(v, o);
    }
    if (lane == 0) finish(O + row, comb<OP>(comb<OP>(v.x, v.z), comb<OP>(v.y, v.w)), acc, mean_div);
  }
}

// The same for short rows (128 ... 1024 columns, S = s known at compile time): a warp works on four
// rows at a time so that the loads of all four are in flight before the first shuffle (one row
// per iteration left the kernel latency-bound at 2.7 TB/s on rows of 256 columns).
template <int OP, int S>
__global__ void __launch_bounds__(kThreads)
reduce_warp4_short_kernel(float* __restrict__ O, const float* __restrict__ I, RedGeom g, Levels L, int acc,
                          float mean_div) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row0 = warp0 * 4; row0 < g.rows; row0 += nwarps * 4) {
    float4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t row = row0 + q < g.rows ? row0 + q : g.rows - 1;      // the tail repeats the last row
      v[q] = subtree_of<OP, float4, S, true>(I + row_base(g, row), 4u * lane, S, L, g);
    }
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float4 o;
        o.x = __shfl_down_sync(0xffffffffu, v[q].x, h); o.y = __shfl_down_sync(0xffffffffu, v[q].y, h);
        o.z = __shfl_down_sync(0xffffffffu, v[q].z, h); o.w = __shfl_down_sync(0xffffffffu, v[q].w, h);
        if (lane < h) v[q] = comb<OP>(v[q], o);
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (row0 + q < g.rows)
          finish(O + row0 + q, comb<OP>(comb<OP>(v[q].x, v[q].z), comb<OP>(v[q].y, v[q].w)), acc, mean_div);
    }
  }
}

// Number of blocks of a single-row reduction that have stored their partials; the block that
// finds itself last finishes the row and resets the counter for the next launch.
static __device__ unsigned int g_blocks_done;

// The halving tree over x[i] = P[first + stride * i], i < m (m a power of two): stage after stage
// element i is combined with element i + m/2.  Leaves are visited in bit-reversed order so that
// a binary-counter stack meets them in exactly that pairing; eight loads are in flight at a time.
// P was written by other blocks of the same launch: the loads go to L2.
template <int OP>
__device__ float strided_halving_tree(const float* P, int64_t first, int64_t stride, int m) {
  float stack[24];
  const int bits = 31 - __clz(m);
  float w = 0.0f;
  for (int k0 = 0; k0 < m; k0 += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u;
      const int i = bits ? (int)(__brev((unsigned)k) >> (32 - bits)) : 0;
      v[u] = k < m ? __ldcg(P + first + stride * i) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u;
      if (k < m) {
        w = v[u];
        int level = 0;
        for (int kk = k; kk & 1; kk >>= 1, ++level) w = comb<OP>(stack[level], w);
        stack[level] = w;
      }
    }
  }
  return w;
}

// One kept row, power-of-two column count, at most 2^14 partials: the last block to arrive runs the
// rest of the same tree over them instead of two more dependent launches.
template <int OP>
__global__ void __launch_bounds__(kThreads, 4)
reduce_single_row_kernel(float* __restrict__ O, float* __restrict__ P, const float* __restrict__ I,
                         RedGeom g, Levels L, int s, int acc, float mean_div) {
  __shared__ float tail_vals[kThreads];
  __shared__ int is_last;
  const int64_t parts = L.n[s];
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < (parts >> 2); gid += nthreads)
    *reinterpret_cast<float4*>(P + (gid << 2)) = subtree<OP, float4>(I, (uint32_t)(gid << 2), s, L, g);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int prev = atomicAdd(&g_blocks_done, 1u);
    is_last = prev == gridDim.x - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  const int width = parts < kThreads ? (int)parts : kThreads;      // a power of two
  if ((int)threadIdx.x < width)
    tail_vals[threadIdx.x] = strided_halving_tree<OP>(P, threadIdx.x, width, (int)(parts / width));
  __syncthreads();
  for (int h = width >> 1; h >= 1; h >>= 1) {
    float nv = 0.0f;
    if ((int)threadIdx.x < h) nv = comb<OP>(tail_vals[threadIdx.x], tail_vals[threadIdx.x + h]);
    __syncthreads();
    if ((int)threadIdx.x < h) tail_vals[threadIdx.x] = nv;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    finish(O, tail_vals[0], acc, mean_div);
    g_blocks_done = 0u;
  }
}

// ---- COLS >= 2^31: the same tree by a depth-first walk with 64-bit indices, one thread per partial ----
struct Levels64 { int S; int64_t n[kMaxLevels + 1]; };
template <int OP>
__global__ void __launch_bounds__(kThreads)
reduce_huge_kernel(float* __restrict__ P, const float* __restrict__ I, RedGeom g, Levels64 L, int s) {
  const int64_t parts = L.n[s], total = g.rows * parts;
  for (int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < total; gid += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = gid / parts, c0 = gid - row * parts;
    const float* base = I + row_base(g, row);
    float acc[kMaxLevels];
    int64_t leaf = c0;
    uint64_t m = 0;
    float v;
    for (;;) {
      const int64_t q = leaf / g.r1;
      v = __ldcs(base + q * g.stride_r0 + (leaf - q * g.r1) * g.stride_r1);
      int64_t cur = leaf;
      int j = 1;
      for (; j <= s; ++j) {
        if ((m >> (j - 1)) & 1ull) {
          v = comb<OP>(acc[j], v);
          cur -= L.n[j];
        } else if (cur + L.n[j] < L.n[j - 1]) {
          acc[j] = v;
          break;
        }
      }
      if (j > s) break;
      m = ((m >> (j - 1)) | 1ull) << (j - 1);
      leaf = cur + L.n[j];
    }
    P[row * parts + c0] = v;
  }
}

// ---- gradients -------------------------------------------------------------------------------
// acc != 0: dI += ..., else dI = ... (every element is written, so a gradient that has not been
// touched yet needs neither a zero fill nor a read).

// Element index of dI -> (row, column) of the reduction.
__device__ __forceinline__ void locate(const RedGeom& g, int64_t x, int64_t& row, int64_t& col) {
  if (g.small) {
    uint32_t v = (uint32_t)x, q = g.by_inner.div(v);
    const uint32_t inner_i = v - q * g.by_inner.d;
    v = q; q = g.by_r1.div(v);
    const uint32_t c1 = v - q * g.by_r1.d;
    v = q; q = g.by_mid.div(v);
    const uint32_t mid_i = v - q * g.by_mid.d;
    v = q; q = g.by_r0.div(v);
    const uint32_t c0 = v - q * g.by_r0.d;
    row = ((int64_t)q * g.by_mid.d + mid_i) * g.by_inner.d + inner_i;
    col = (int64_t)c0 * g.by_r1.d + c1;
    return;
  }
  const int64_t inner_i = x % g.inner; x /= g.inner;
  const int64_t c1 = x % g.r1; x /= g.r1;
  const int64_t mid_i = x % g.mid; x /= g.mid;
  const int64_t c0 = x % g.r0; x /= g.r0;
  row = (x * g.mid + mid_i) * g.inner + inner_i;
  col = c0 * g.r1 + c1;
}

// dI (+)= dO[row] (/ COLS)   (reduce.py:250-260).  V = float4: four consecutive elements share a row
// (inner == 1, r1 % 4 == 0) or every index but the innermost (inner % 4 == 0: dO is read as float4 too).
template <class V>
__global__ void __launch_bounds__(kThreads)
reduce_bwd_bcast_kernel(float* __restrict__ dI, const float* __restrict__ dO, int64_t total,
                        RedGeom g, float mean_div, int acc) {
  constexpr int VW = sizeof(V) / 4;
  const int64_t tid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VW;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x * VW;
  for (int64_t i = tid; i < total; i += nthreads) {
    int64_t row, col;
    locate(g, i, row, col);
    if (VW == 1) {
      float v = __ldg(dO + row);
      if (mean_div != 0.0f) v = __fdiv_rn(v, mean_div);
      dI[i] = __fadd_rn(acc ? dI[i] : 0.0f, v);
    } else {
      float4 v;
      if (g.inner == 1) { v.x = __ldg(dO + row); v.y = v.z = v.w = v.x; }
      else v = __ldg(reinterpret_cast<const float4*>(dO + row));
      if (mean_div != 0.0f) {
        v.x = __fdiv_rn(v.x, mean_div); v.y = __fdiv_rn(v.y, mean_div);
        v.z = __fdiv_rn(v.z, mean_div); v.w = __fdiv_rn(v.w, mean_div);
      }
      float4* dst = reinterpret_cast<float4*>(dI + i);
      const float4 o = acc ? *dst : make_float4(0.f, 0.f, 0.f, 0.f);
      __stcs(dst, comb<LNN_RED_SUM>(o, v));
    }
  }
}

// max/min: the gradient goes to the lowest column whose value equals the reduced value
// (reduce.py:262-276 gives it to whichever work-item wins an atomic; on tie-free data
// both agree).  Three forms:
//  * select: one thread per row walks its columns and stops at the first match.  Reads half of I and
//    touches one element of dI per row: for "+=" with many rows that are adjacent in memory.
//  * find + put: every element of I is looked at once, by neighbouring threads; matches meet in an
//    atomicMin per row (a few per row, so no contention), and for "=" the same pass writes the zeros of
//    dI; the second launch adds dO at the columns found.  A row as long as the tensor keeps the whole
//    GPU busy, where one thread per row took 1 s on 134 M columns.
__global__ void __launch_bounds__(kThreads)
reduce_bwd_select_kernel(float* __restrict__ dI, const float* __restrict__ I,
                         const float* __restrict__ dO, const float* __restrict__ O, RedGeom g) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t row = tid; row < g.rows; row += nthreads) {
    const int64_t base = row_base(g, row);
    const float o = O[row];
    bool done = false;
    for (int64_t q = 0; q < g.r0 && !done; ++q)
      for (int64_t c = 0; c < g.r1; ++c) {
        const int64_t off = base + q * g.stride_r0 + c * g.stride_r1;
        if (I[off] == o) {
          dI[off] = __fadd_rn(dI[off], dO[row]);
          done = true;
          break;
        }
      }
  }
}

template <class V>
__global__ void __launch_bounds__(kThreads)
reduce_bwd_find_kernel(unsigned long long* __restrict__ first, float* __restrict__ dI, const float* __restrict__ I,
                       const float* __restrict__ O, int64_t total, RedGeom g, int acc) {
  constexpr int VW = sizeof(V) / 4;
  const int64_t tid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VW;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x * VW;
  for (int64_t i = tid; i < total; i += nthreads) {
    int64_t row, col;
    locate(g, i, row, col);
    V v;
    load_leaf(v, I + i);
    const float* e = reinterpret_cast<const float*>(&v);
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      const int64_t r = g.inner == 1 ? row : row + k;
      if (e[k] == __ldg(O + r)) atomicMin(first + r, (unsigned long long)(g.inner == 1 ? col + k : col));
    }
    if (!acc) {
      set_zero(v);
      __stcs(reinterpret_cast<V*>(dI + i), v);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
reduce_bwd_put_kernel(float* __restrict__ dI, const float* __restrict__ dO, const unsigned long long* __restrict__ first,
                      RedGeom g) {
  for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < g.rows; row += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long c = first[row];
    if (c == ~0ull) continue;                       // a NaN row: nothing equals it
    const int64_t q = (int64_t)c / g.r1;
    const int64_t off = row_base(g, row) + q * g.stride_r0 + ((int64_t)c - q * g.r1) * g.stride_r1;
    dI[off] = __fadd_rn(dI[off], dO[row]);
  }
}

int make_geom(RedGeom& g, int64_t outer, int64_t r0, int64_t mid, int64_t r1, int64_t inner) {
  LNN_REQUIRE(outer >= 1 && r0 >= 1 && mid >= 1 && r1 >= 1 && inner >= 1, "bad reduce extents");
  g.outer = outer; g.r0 = r0; g.mid = mid; g.r1 = r1; g.inner = inner;
  g.rows = outer * mid * inner;
  g.stride_r1 = inner;
  g.stride_mid = r1 * inner;
  g.stride_r0 = mid * r1 * inner;
  g.stride_outer = r0 * mid * r1 * inner;
  g.small = outer * g.stride_outer < (1ll << 31);
  if (r1 < (1ll << 31)) g.by_r1 = FastDiv((uint32_t)r1);
  if (g.small) {
    g.by_r0 = FastDiv((uint32_t)r0); g.by_mid = FastDiv((uint32_t)mid); g.by_inner = FastDiv((uint32_t)inner);
  }
  return LNN_OK;
}

void make_levels(Levels& L, uint32_t cols) {
  L.n[0] = cols;
  int s = 0;
  while (L.n[s] > 1) {
    L.n[s + 1] = (L.n[s] + 1) / 2;
    ++s;
  }
  L.S = s;
  L.pow2 = (cols & (cols - 1)) == 0;
  L.exact = 0;
  while (L.exact < s && L.n[L.exact] % 2 == 0) ++L.exact;
  for (int j = s + 1; j <= kMaxLevels; ++j) L.n[j] = 1;
}

inline int grid_for(const lnn::Device* d, int64_t work_items) {
  int64_t blocks = lnn_ceil_div(work_items, kThreads);
  int64_t cap = (int64_t)d->sm_count * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

// Where the partial values of split rows live: pooled memory (lnn_reduce) or a caller-given
// fixed region (lnn_reduce_noalloc).
struct PartialSpace {
  lnn::Device* d;
  float* fixed = nullptr;       // non-null: bump-allocate from [fixed, fixed + cap)
  int64_t cap = 0;
  std::vector<std::pair<void*, uint64_t>> pooled;
  explicit PartialSpace(lnn::Device* dev) : d(dev) {}
  ~PartialSpace() { for (auto& b : pooled) lnn::free_bytes(d, b.first, b.second); }
  int get(int64_t floats, float** out) {
    if (fixed) {
      const int64_t need = (floats + 63) & ~63ll;
      if (need > cap)
        return lnn::set_error(LNN_E_UNSUPPORTED,
                              "reduction needs %lld more floats of scratch but the static scratch has %lld "
                              "left (1 MiB in total): use lnn_reduce", (long long)need, (long long)cap);
      *out = fixed; fixed += need; cap -= need;
      return LNN_OK;
    }
    void* p = nullptr;
    int rc = lnn::alloc_bytes(d, (uint64_t)floats * 4, &p);
    if (rc) return rc;
    pooled.push_back({p, (uint64_t)floats * 4});
    *out = (float*)p;
    return LNN_OK;
  }
};

inline bool aligned16(const void* p) { return (((uintptr_t)p) & 15) == 0; }

// Rows of at most 256 columns (eight where inner > 1): up to eight leaves per lane and as many lanes per row as
// that takes; with inner > 1 one lane per row, whose loads coalesce as they are.  A warp per row whatever its length
// leaves most lanes idle, and the general subtree issues sixteen predicated loads for two or three columns.
// us, those -> here, 16 M elements in rows of 1, 3, 8, 64, 100 columns: 8234 -> 58, 2944 -> 25, 1118 -> 21,
// 168 -> 25, 126 -> 36.  [n, c, 7] over axis 1, 8 M elements, c = 2, 4, 8: 90 -> 15, 52 -> 13, 36 -> 13.
template <int OP>
int launch_rows(lnn::Device* d, float* O, const float* I, const RedGeom& g, const Levels& L, int acc, float mean_div) {
  int w = 1;
  if (g.inner == 1) while (L.n[0] > 8u * w) w <<= 1;
  int s = 0;
  while ((int)L.n[s] > w) ++s;                           // s == 3 wherever w > 1
  const int64_t blocks = std::min<int64_t>(lnn_ceil_div(g.rows, kThreads / w), (int64_t)d->sm_count * 16);
#define CASE(W, S)                                                                                              \
  case (W) * 8 + (S): reduce_rows_kernel<OP, W, S><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, acc, mean_div); break
  switch (w * 8 + s) {
    CASE(1, 0); CASE(1, 1); CASE(1, 2); CASE(1, 3);
    CASE(2, 3); CASE(4, 3); CASE(8, 3); CASE(16, 3); CASE(32, 3);
    default: return lnn::set_error(LNN_E_UNSUPPORTED, "rows of %u columns are not short", L.n[0]);
  }
#undef CASE
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

// Plans one reduction as 1..3 launches.  mean_div is the ORIGINAL column count (as float)
// for mean, 0 otherwise; it is applied only where a row is finished.
template <int OP>
int reduce_impl(lnn::Device* d, PartialSpace& space, float* O, const float* I, int64_t outer,
                int64_t r0, int64_t mid, int64_t r1, int64_t inner, int acc, float mean_div) {
  RedGeom g;
  int rc = make_geom(g, outer, r0, mid, r1, inner);
  if (rc) return rc;
  const int64_t cols = r0 * r1;
  if (cols >= (1ll << 31)) {
    Levels64 L;
    L.S = 0; L.n[0] = cols;
    while (L.n[L.S] > 1) { L.n[L.S + 1] = (L.n[L.S] + 1) / 2; ++L.S; }
    int s = 9;
    while (s < L.S && g.rows * L.n[s] > (1 << 24)) ++s;
    float* part = nullptr;
    rc = space.get(g.rows * L.n[s], &part);
    if (rc) return rc;
    reduce_huge_kernel<OP><<<grid_for(d, g.rows * L.n[s]), kThreads, 0, d->stream>>>(part, I, g, L, s);
    LNN_CHECK_LAUNCH(d);
    return reduce_impl<OP>(d, space, O, part, g.rows, 1, 1, L.n[s], 1, acc, mean_div);
  }
  Levels L;
  make_levels(L, (uint32_t)cols);
  const int64_t kTargetThreads = 1 << 19;
  const int64_t sms = d->sm_count;
  if (inner == 1) {
    // Rows too few to give every SM several blocks and long enough to pay for a second launch are
    // split over many threads first.
    const bool split = (g.rows * kThreads < kTargetThreads / 2 && cols >= 16384) ||
                       (g.rows == 1 && L.pow2 && cols >= 8192);
    // 128-bit loads of four adjacent columns need contiguous, 16-byte aligned columns
    const bool cols_vec = aligned16(I) && (r0 == 1 || (r1 % 4 == 0 && g.stride_r0 % 4 == 0)) &&
                          g.stride_mid % 4 == 0 && g.stride_outer % 4 == 0;
    if (!split) {
      // one warp per row as soon as the rows fill the GPU with warps; a block's worth of threads per
      // row below that (a warp would be a single latency-bound chain)
      const bool enough_warps = g.rows >= sms * 16 || cols <= 512;
      if (enough_warps && L.pow2 && cols_vec && cols >= 128) {
        const int s = L.S - 7;                           // 128 partials per row, four per lane
        const int64_t cap = sms * 16;
        int64_t blocks = std::min<int64_t>(lnn_ceil_div(g.rows, kThreads / 32), cap);
        if (s <= 3 && g.rows >= 4096) {
          blocks = std::min<int64_t>(lnn_ceil_div(g.rows, 4 * (kThreads / 32)), cap);
          switch (s) {
            case 0: reduce_warp4_short_kernel<OP, 0><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, acc, mean_div); break;
            case 1: reduce_warp4_short_kernel<OP, 1><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, acc, mean_div); break;
            case 2: reduce_warp4_short_kernel<OP, 2><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, acc, mean_div); break;
            default: reduce_warp4_short_kernel<OP, 3><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, acc, mean_div); break;
          }
        } else {
          reduce_warp4_kernel<OP><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, s, acc, mean_div);
        }
        LNN_CHECK_LAUNCH(d);
        return LNN_OK;
      }
      if (cols <= 256) return launch_rows<OP>(d, O, I, g, L, acc, mean_div);
      if (enough_warps) {
        int s = 0;
        while (L.n[s] > 32) ++s;
        const int64_t blocks = std::min<int64_t>(lnn_ceil_div(g.rows, kThreads / 32), sms * 16);
        reduce_warp_kernel<OP><<<(unsigned)blocks, kThreads, 0, d->stream>>>(O, I, g, L, s, acc, mean_div);
        LNN_CHECK_LAUNCH(d);
        return LNN_OK;
      }
      int s_block = 0;                       // smallest s with n[s] <= 256
      while (L.n[s_block] > kThreads) ++s_block;
      int tpr = 1;
      while (tpr < (int)L.n[s_block]) tpr <<= 1;
      const int64_t blocks = lnn_ceil_div(g.rows, kThreads / tpr);
      LNN_REQUIRE(blocks < (1ll << 31), "too many rows");
      reduce_rowcoop_kernel<OP><<<(unsigned)blocks, kThreads, 0, d->stream>>>(
          O, I, g, L, s_block, tpr, acc, mean_div);
      LNN_CHECK_LAUNCH(d);
      return LNN_OK;
    }
    // enough threads to fill the GPU (a 128-bit thread covers four partials), at least 16 leaves each
    int s_vec = 0;                           // stages over which four adjacent columns stay together
    while (cols_vec && s_vec < L.exact && L.n[s_vec + 1] % 4 == 0) ++s_vec;
    const bool vec = s_vec >= 3;
    int64_t target_vals = vec ? 4 * kTargetThreads / 2 : kTargetThreads;
    if (space.fixed) target_vals = std::min<int64_t>(target_vals, std::max<int64_t>(space.cap / 2, 1024));
    int s = L.pow2 ? 6 : 4;
    while (s < L.S && g.rows * L.n[s] > target_vals) ++s;
    if (L.pow2 && s > kMaxPow2Levels) s = kMaxPow2Levels;
    // A single row of a few hundred thousand columns (the partials of an all-axes reduction): 16
    // leaves per thread and at most 2^14 partials, which the last block of the same launch finishes.
    const bool finish_here = g.rows == 1 && L.pow2 && cols_vec && cols <= (1ll << 18) && cols >= (1ll << 12);
    if (finish_here) s = 4;
    const bool vec_now = vec && (!space.fixed || s <= s_vec);
    if (vec_now && s > s_vec) s = s_vec;
    const int64_t parts = L.n[s];
    float* part = nullptr;
    rc = space.get(g.rows * parts, &part);
    if (rc) return rc;
    // the partials of one kept row are stored contiguously, [row][parts], whatever the position of
    // the kept axes: the second pass is then a plain row reduction over `parts` columns, the tail
    // of the same tree
    if (finish_here) {
      reduce_single_row_kernel<OP><<<grid_for(d, parts / 4), kThreads, 0, d->stream>>>(O, part, I, g, L, s, acc, mean_div);
      LNN_CHECK_LAUNCH(d);
      return LNN_OK;
    }
    if (vec_now && aligned16(part))
      reduce_parts_kernel<OP, float4><<<grid_for(d, g.rows * parts / 4), kThreads, 0, d->stream>>>(
          nullptr, part, I, g, L, s, 1, 0, 0.0f);
    else
      reduce_parts_kernel<OP, float><<<grid_for(d, g.rows * parts), kThreads, 0, d->stream>>>(
          nullptr, part, I, g, L, s, 1, 0, 0.0f);
    LNN_CHECK_LAUNCH(d);
    return reduce_impl<OP>(d, space, O, part, g.rows, 1, 1, parts, 1, acc, mean_div);
  }
  // inner > 1: coalesce along the inner axis; four adjacent kept rows per thread when it allows 128-bit loads
  const bool vec = inner % 4 == 0 && aligned16(I) && aligned16(O);
  const int64_t groups = g.rows / (vec ? 4 : 1);         // columns of threads
  if (!vec && cols <= 8 && groups >= sms * kThreads) return launch_rows<OP>(d, O, I, g, L, acc, mean_div);
  if (cols <= (vec ? 16 : 32) && groups >= sms * kThreads) {
    // short columns, many of them: one thread each.  (With scalar loads the block kernel's stages cost more up
    // to 32 columns: [n, 17, 7] and [n, 32, 7], 8 M elements, 37 and 23 us there, 32 and 12 here.)
    if (vec)
      reduce_parts_kernel<OP, float4><<<grid_for(d, groups), kThreads, 0, d->stream>>>(O, nullptr, I, g, L, L.S, 0, acc, mean_div);
    else
      reduce_parts_kernel<OP, float><<<grid_for(d, groups), kThreads, 0, d->stream>>>(O, nullptr, I, g, L, L.S, 0, acc, mean_div);
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  const int64_t col_blocks = lnn_ceil_div(groups, 32);
  // Long columns with too few blocks to cover the SMs twice are split over a first pass; up to 32
  // leaves per thread the block kernel's one launch is shorter than two.
  const bool split = col_blocks < 2 * sms && lnn_ceil_div(cols, kColParts) > 32;
  if (!split) {
    int s = 0;
    while ((int)L.n[s] > kColParts) ++s;
    const unsigned blocks = (unsigned)std::min<int64_t>(col_blocks, 1 << 30);
    if (vec)
      reduce_cols_kernel<OP, float4><<<blocks, kThreads, 0, d->stream>>>(O, I, g, L, s, acc, mean_div);
    else
      reduce_cols_kernel<OP, float><<<blocks, kThreads, 0, d->stream>>>(O, I, g, L, s, acc, mean_div);
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  int64_t target_vals = vec ? 4 * kTargetThreads / 2 : kTargetThreads;
  if (space.fixed) target_vals = std::min<int64_t>(target_vals, std::max<int64_t>(space.cap / 2, 1024));
  int s = 4;
  while (s < L.S && g.rows * L.n[s] > target_vals) ++s;
  const int64_t parts = L.n[s];
  float* part = nullptr;
  rc = space.get(g.rows * parts, &part);
  if (rc) return rc;
  if (parts == 1) part = O;                              // (only a bounded scratch drives s that far)
  if (vec && aligned16(part))
    reduce_parts_kernel<OP, float4><<<grid_for(d, groups * parts), kThreads, 0, d->stream>>>(
        parts == 1 ? O : nullptr, part, I, g, L, s, 0, parts == 1 ? acc : 0, parts == 1 ? mean_div : 0.0f);
  else
    reduce_parts_kernel<OP, float><<<grid_for(d, g.rows * parts), kThreads, 0, d->stream>>>(
        parts == 1 ? O : nullptr, part, I, g, L, s, 0, parts == 1 ? acc : 0, parts == 1 ? mean_div : 0.0f);
  LNN_CHECK_LAUNCH(d);
  if (parts == 1) return LNN_OK;
  return reduce_impl<OP>(d, space, O, part, outer, parts, 1, 1, mid * inner, acc, mean_div);
}

// dI (+)= the gradient of a reduction; `accumulate` as above.
int reduce_bwd(lnn::Device* d, int op, uint64_t dI, uint64_t I, uint64_t dO, uint64_t O, int64_t outer,
               int64_t r0, int64_t mid, int64_t r1, int64_t inner, int acc) {
  RedGeom g;
  int rc = make_geom(g, outer, r0, mid, r1, inner);
  if (rc) return rc;
  const int64_t total = g.rows * r0 * r1;
  float* di = (float*)(uintptr_t)dI;
  const float* dout = (const float*)(uintptr_t)dO;
  const bool together = inner % 4 == 0 || (inner == 1 && r1 % 4 == 0);   // four elements of one row, or of four
  if (op == LNN_RED_SUM || op == LNN_RED_MEAN) {
    const float mean_div = op == LNN_RED_MEAN ? (float)(r0 * r1) : 0.0f;
    if (together && (dI & 15) == 0 && (inner == 1 || (dO & 15) == 0))
      reduce_bwd_bcast_kernel<float4><<<grid_for(d, total / 4), kThreads, 0, d->stream>>>(di, dout, total, g, mean_div, acc);
    else
      reduce_bwd_bcast_kernel<float><<<grid_for(d, total), kThreads, 0, d->stream>>>(di, dout, total, g, mean_div, acc);
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  if (op != LNN_RED_MAX && op != LNN_RED_MIN) return lnn::set_error(LNN_E_INVALID, "unknown reduce op %d", op);
  LNN_REQUIRE(I && O, "max/min backward needs I and O");
  const float* in = (const float*)(uintptr_t)I;
  const float* out = (const float*)(uintptr_t)O;
  if (acc && inner >= 32 && g.rows >= (int64_t)d->sm_count * kThreads) {
    reduce_bwd_select_kernel<<<grid_for(d, g.rows), kThreads, 0, d->stream>>>(di, in, dout, out, g);
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  lnn::Scratch first(d);
  rc = first.get((uint64_t)g.rows * 8);
  if (rc) return rc;
  LNN_CUDA(cudaMemsetAsync(first.p, 0xff, (size_t)g.rows * 8, d->stream));
  if (together && ((dI | I) & 15) == 0)
    reduce_bwd_find_kernel<float4><<<grid_for(d, total / 4), kThreads, 0, d->stream>>>(
        first.as<unsigned long long>(), di, in, out, total, g, acc);
  else
    reduce_bwd_find_kernel<float><<<grid_for(d, total), kThreads, 0, d->stream>>>(
        first.as<unsigned long long>(), di, in, out, total, g, acc);
  LNN_CHECK_LAUNCH(d);
  reduce_bwd_put_kernel<<<grid_for(d, g.rows), kThreads, 0, d->stream>>>(di, dout, first.as<unsigned long long>(), g);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int reduce_dispatch(lnn::Device* d, PartialSpace& space, int op, uint64_t O, uint64_t I, int64_t outer,
                    int64_t r0, int64_t mid, int64_t r1, int64_t inner, int accumulate) {
  float* o = (float*)(uintptr_t)O;
  const float* i = (const float*)(uintptr_t)I;
  const float cols_f = (float)(r0 * r1);
  switch (op) {
    case LNN_RED_SUM: return reduce_impl<LNN_RED_SUM>(d, space, o, i, outer, r0, mid, r1, inner, accumulate, 0.0f);
    case LNN_RED_MEAN: return reduce_impl<LNN_RED_SUM>(d, space, o, i, outer, r0, mid, r1, inner, accumulate, cols_f);
    case LNN_RED_MAX: return reduce_impl<LNN_RED_MAX>(d, space, o, i, outer, r0, mid, r1, inner, accumulate, 0.0f);
    case LNN_RED_MIN: return reduce_impl<LNN_RED_MIN>(d, space, o, i, outer, r0, mid, r1, inner, accumulate, 0.0f);
  }
  return lnn::set_error(LNN_E_INVALID, "unknown reduce op %d", op);
}

// ---- reduction without any allocation ---------------------------------------------------------
// Partial results of split rows live in this fixed device array instead of pooled memory.
// Every device that loads the library holds its own 1 MiB copy until the process exits.
constexpr int64_t kStaticScratchFloats = 1 << 18;
static __device__ __align__(256) float g_static_scratch[kStaticScratchFloats];

// Device address of g_static_scratch per device slot, resolved once per device.  In host
// code the symbol itself is only a stand-in; kernels must be given this address.
float* g_static_scratch_ptr[LNN_MAX_DEVICES] = {nullptr};

int static_scratch_for(lnn::Device* d, int dev, float** out) {
  if (!g_static_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);   // d's device is current
    if (e != cudaSuccess || !p)
      return lnn::set_error(LNN_E_CUDA, "cudaGetSymbolAddress(static scratch) failed on device %d: %s",
                            d->ordinal, cudaGetErrorString(e));
    g_static_scratch_ptr[dev] = (float*)p;
  }
  *out = g_static_scratch_ptr[dev];
  return LNN_OK;
}

}  // namespace

extern "C" {

int lnn_reduce(int dev, int op, uint64_t O, uint64_t I, int64_t outer, int64_t r0, int64_t mid,
               int64_t r1, int64_t inner, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(O && I, "null buffer");
  LNN_REQUIRE(outer >= 1 && r0 >= 1 && mid >= 1 && r1 >= 1 && inner >= 1, "bad reduce extents");
  PartialSpace space(d);
  return reduce_dispatch(d, space, op, O, I, outer, r0, mid, r1, inner, accumulate);
}

int lnn_reduce_bwd(int dev, int op, uint64_t dI, uint64_t I, uint64_t dO, uint64_t O, int64_t outer,
                   int64_t r0, int64_t mid, int64_t r1, int64_t inner) {
  return lnn_reduce_bwd_acc(dev, op, dI, I, dO, O, outer, r0, mid, r1, inner, 1);
}

int lnn_reduce_bwd_acc(int dev, int op, uint64_t dI, uint64_t I, uint64_t dO, uint64_t O, int64_t outer,
                       int64_t r0, int64_t mid, int64_t r1, int64_t inner, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dI && dO, "null buffer");
  return reduce_bwd(d, op, dI, I, dO, O, outer, r0, mid, r1, inner, accumulate);
}

// Reduction for callers that must not allocate device memory: a host thread inside a
// latency-critical serving loop, a library embedded in an application that has handed the
// whole GPU heap to its own allocator, or code running after memory has been exhausted --
// cudaMalloc there either stalls the device or fails.  Same arguments and bit-identical
// results as lnn_reduce; the partial sums of rows that are split across thread blocks are
// kept in a fixed 1 MiB device array that belongs to the library (one copy per device,
// held until the process exits) instead of pooled memory.
//  * Reductions whose partials do not fit (more than 2^18 floats) are refused with
//    LNN_E_UNSUPPORTED; nothing more is launched once that is found.
//  * The first call on a device resolves the array's device address (one
//    cudaGetSymbolAddress, no allocation); make that first call before any stream capture.
//  * All calls share the one array and it keeps whatever the previous call left; every
//    partial a launch reads has been written by the launch before it, so nothing needs
//    clearing.  Calls follow each other on the device's single stream; two calls made to
//    overlap on the GPU (by driving the same device from two threads) would race on it.
int lnn_reduce_noalloc(int dev, int op, uint64_t O, uint64_t I, int64_t outer, int64_t r0, int64_t mid,
                       int64_t r1, int64_t inner, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(O && I, "null buffer");
  LNN_REQUIRE(outer >= 1 && r0 >= 1 && mid >= 1 && r1 >= 1 && inner >= 1, "bad reduce extents");
  float* scratch = nullptr;
  int rc = static_scratch_for(d, dev, &scratch);
  if (rc) return rc;
  PartialSpace space(d);
  space.fixed = scratch;
  space.cap = kStaticScratchFloats;
  return reduce_dispatch(d, space, op, O, I, outer, r0, mid, r1, inner, accumulate);
}

}  // extern "C"
