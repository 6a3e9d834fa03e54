// 2-D pooling forward/backward (avg, max, min) on NCHW fp32.
// Semantics follow litenn/core/op/pool2D.py:111-230: taps are visited in row-major
// window order; avg divides the ordered sum by the number of in-bounds taps; max/min of
// an empty window is 0; the max/min gradient goes to the FIRST tap (row-major) equal to
// the pooled value.  HBM-bound: the 2x2/stride-2 even-width case reads two float4 rows
// per two outputs and writes float2; everything else uses the generic kernels, which clip each
// window to the image once instead of testing every tap.
#include "lnn_common.cuh"
#include <math_constants.h>

namespace {

constexpr int kThreads = 256;

struct PoolGeom {
  int ih, iw, oh, ow, pool, stride, padl, padt;
  lnn::FastDiv by_iw, by_ih, by_ow, by_oh, by_stride;
  PoolGeom(int ih_, int iw_, int oh_, int ow_, int pool_, int stride_, int padl_, int padt_)
      : ih(ih_), iw(iw_), oh(oh_), ow(ow_), pool(pool_), stride(stride_), padl(padl_), padt(padt_),
        by_iw((uint32_t)iw_), by_ih((uint32_t)ih_), by_ow((uint32_t)ow_), by_oh((uint32_t)oh_), by_stride((uint32_t)stride_) {}
};

// index -> (plane, row, column) of a tensor of rows x cols planes
__device__ __forceinline__ void split_index(int64_t i, const lnn::FastDiv& by_cols, const lnn::FastDiv& by_rows,
                                            int64_t& plane, int& row, int& col) {
  if (i < (1ll << 31)) {
    const uint32_t r = by_cols.div((uint32_t)i), p = by_rows.div(r);
    col = (int)((uint32_t)i - r * by_cols.d); row = (int)(r - p * by_rows.d); plane = p;
  } else {
    const int64_t r = i / by_cols.d;
    plane = r / by_rows.d; col = (int)(i - r * by_cols.d); row = (int)(r - plane * by_rows.d);
  }
}

constexpr uint8_t kNoWinner = 255;     // a window none of whose elements equals its pooled value (NaN, empty)

// The part of window (oh, ow) that lies inside the image: rows [h0, h1), columns [w0, w1).
struct Window { int h0, h1, w0, w1; };
__device__ __forceinline__ Window window_of(const PoolGeom& g, int oh, int ow) {
  Window w;
  const int top = oh * g.stride - g.padt, left = ow * g.stride - g.padl;
  w.h0 = max(top, 0); w.h1 = min(top + g.pool, g.ih);
  w.w0 = max(left, 0); w.w1 = min(left + g.pool, g.iw);
  return w;
}

// Generic forward: one thread per output.  The window is clipped to the image once, then its
// elements are combined in row-major order, which is the order in which the reference visits
// the taps it does not skip (pool2D.py:111-146): sum / (number of in-image taps), or max / min
// with 0 for a window that lies entirely outside.  idx (max / min, optional) receives the place of
// the first element equal to the pooled value, row * pool + column within the unclipped window, which
// is where the gradient goes.
template <int MODE>
__global__ void __launch_bounds__(kThreads)
pool_fwd_kernel(float* __restrict__ O, uint8_t* __restrict__ idx, const float* __restrict__ I, int64_t total, const PoolGeom g) {
  for (int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < total; gid += (int64_t)gridDim.x * blockDim.x) {
    int64_t pl;
    int oh, ow;
    split_index(gid, g.by_ow, g.by_oh, pl, oh, ow);
    const float* plane = I + pl * g.ih * g.iw;
    const Window w = window_of(g, oh, ow);
    const float start = MODE == LNN_POOL_AVG ? 0.0f : (MODE == LNN_POOL_MAX ? -CUDART_INF_F : CUDART_INF_F);
    float acc = start;
    int first = -1;                                   // place of the element acc came from
    const int top = oh * g.stride - g.padt, left = ow * g.stride - g.padl;
    for (int h = w.h0; h < w.h1; ++h) {
      const float* row = plane + (int64_t)h * g.iw;
      for (int x = w.w0; x < w.w1; ++x) {
        const float v = row[x];
        if (MODE == LNN_POOL_AVG) acc = __fadd_rn(acc, v);
        else {
          // (an element equal to the running value is not an earlier one; +-0 compare equal, as in the gradient)
          if (MODE == LNN_POOL_MAX ? v > acc : v < acc) first = (h - top) * g.pool + (x - left);
          else if (first < 0 && v == acc) first = (h - top) * g.pool + (x - left);
          acc = MODE == LNN_POOL_MAX ? fmaxf(acc, v) : fminf(acc, v);
        }
      }
    }
    const int count = max(w.h1 - w.h0, 0) * max(w.w1 - w.w0, 0);
    if (MODE == LNN_POOL_AVG) { if (count > 0) acc = __fdiv_rn(acc, (float)count); }
    else if (acc == start) { acc = 0.0f; first = -1; }   // the stored 0 replaces the infinity the window holds
    O[gid] = acc;
    if (MODE != LNN_POOL_AVG && idx) idx[gid] = first < 0 ? kNoWinner : (uint8_t)first;
  }
}

// 2x2 / stride 2 / no left-top padding / even IW, OW == IW/2: a thread produces NW horizontally
// adjacent outputs from two vectors of 2 * NW elements (NW = 2 when IW is a multiple of 4).  All taps in
// bounds except possibly the bottom row when IH is odd (padded bottom).  idx: as above, 0..3; without IDX nothing
// looks for the winner (128 x 128 x 112 x 112: 159 us when a null map was left out at run time, 152 so).
template <int NW> struct PoolVec;
template <> struct PoolVec<2> { typedef float4 In; typedef float2 Out; typedef uchar2 Idx; };
template <> struct PoolVec<1> { typedef float2 In; typedef float Out; typedef uint8_t Idx; };

template <int MODE, int NW, bool IDX>
__global__ void __launch_bounds__(kThreads)
pool2x2_fwd_kernel(float* __restrict__ O, uint8_t* __restrict__ idx, const float* __restrict__ I, int64_t total, int ih,
                   int iw, lnn::FastDiv by_ow, lnn::FastDiv by_oh) {
  typedef typename PoolVec<NW>::In In;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < total; gid += nthreads) {
    int64_t plane;
    int y, xq;
    split_index(gid, by_ow, by_oh, plane, y, xq);                   // by_ow counts groups of NW outputs
    const float* row0 = I + (plane * ih + 2 * y) * (int64_t)iw + 2 * NW * xq;
    __align__(16) float a[2 * NW];
    __align__(16) float b[2 * NW];
    __align__(16) float r[NW];
    __align__(4) uint8_t w[NW];
    *reinterpret_cast<In*>(a) = __ldcs(reinterpret_cast<const In*>(row0));
    const bool has1 = (2 * y + 1) < ih;
    if (has1) *reinterpret_cast<In*>(b) = __ldcs(reinterpret_cast<const In*>(row0 + iw));
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const float t0 = a[2 * k], t1 = a[2 * k + 1];
      if (MODE == LNN_POOL_AVG) {
        // ordered sum ((0 + t00) + t01) + t10) + t11 ; 0 + t00 == t00 except for -0
        float s = __fadd_rn(__fadd_rn(0.0f, t0), t1);
        if (has1) s = __fadd_rn(__fadd_rn(s, b[2 * k]), b[2 * k + 1]);
        r[k] = __fdiv_rn(s, has1 ? 4.0f : 2.0f);
        continue;
      }
      const float start = MODE == LNN_POOL_MAX ? -CUDART_INF_F : CUDART_INF_F;
      float m = MODE == LNN_POOL_MAX ? fmaxf(fmaxf(start, t0), t1) : fminf(fminf(start, t0), t1);
      if (has1) m = MODE == LNN_POOL_MAX ? fmaxf(fmaxf(m, b[2 * k]), b[2 * k + 1]) : fminf(fminf(m, b[2 * k]), b[2 * k + 1]);
      if (m == start) m = 0.0f;
      r[k] = m;
      if (IDX) w[k] = t0 == m ? 0 : t1 == m ? 1 : has1 && b[2 * k] == m ? 2 : has1 && b[2 * k + 1] == m ? 3 : kNoWinner;
    }
    __stcs(reinterpret_cast<typename PoolVec<NW>::Out*>(O) + gid, *reinterpret_cast<typename PoolVec<NW>::Out*>(r));
    if (IDX)
      reinterpret_cast<typename PoolVec<NW>::Idx*>(idx)[gid] = *reinterpret_cast<typename PoolVec<NW>::Idx*>(w);
  }
}

// Gradient of the same case from the map of winners (MODE max, which serves min too) or of the average:
// neither the input nor the output is read again.  64 x 128 x 112 x 112: 162 us with both re-read, 85 us here.
template <int MODE, int NW>
__global__ void __launch_bounds__(kThreads)
pool2x2_bwd_idx_kernel(float* __restrict__ dI, const uint8_t* __restrict__ idx, const float* __restrict__ dO, int64_t total,
                       int ih, int iw, lnn::FastDiv by_ow, lnn::FastDiv by_oh, int acc) {
  typedef typename PoolVec<NW>::In In;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < total; gid += nthreads) {
    int64_t plane;
    int y, xq;
    split_index(gid, by_ow, by_oh, plane, y, xq);
    float* row0 = dI + (plane * ih + 2 * y) * (int64_t)iw + 2 * NW * xq;
    const bool has1 = (2 * y + 1) < ih;
    __align__(16) float g[NW];
    __align__(16) float a[2 * NW];
    __align__(16) float b[2 * NW];
    __align__(4) uint8_t w[NW];
    *reinterpret_cast<typename PoolVec<NW>::Out*>(g) = __ldcs(reinterpret_cast<const typename PoolVec<NW>::Out*>(dO) + gid);
    if (MODE != LNN_POOL_AVG)
      *reinterpret_cast<typename PoolVec<NW>::Idx*>(w) = __ldcs(reinterpret_cast<const typename PoolVec<NW>::Idx*>(idx) + gid);
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      // the reference adds 0.0 + dO to its accumulator first, then accumulator to dI
      const float u = __fadd_rn(0.0f, MODE == LNN_POOL_AVG ? __fdiv_rn(g[k], has1 ? 4.0f : 2.0f) : g[k]);
      if (MODE == LNN_POOL_AVG) a[2 * k] = a[2 * k + 1] = b[2 * k] = b[2 * k + 1] = u;
      else {
        a[2 * k] = w[k] == 0 ? u : 0.0f; a[2 * k + 1] = w[k] == 1 ? u : 0.0f;
        b[2 * k] = w[k] == 2 ? u : 0.0f; b[2 * k + 1] = w[k] == 3 ? u : 0.0f;
      }
    }
    __align__(16) float o[2 * NW];
    if (acc) {
      *reinterpret_cast<In*>(o) = *reinterpret_cast<const In*>(row0);
#pragma unroll
      for (int k = 0; k < 2 * NW; ++k) a[k] = __fadd_rn(o[k], a[k]);
    }
    __stcs(reinterpret_cast<In*>(row0), *reinterpret_cast<In*>(a));
    if (has1) {
      if (acc) {
        *reinterpret_cast<In*>(o) = *reinterpret_cast<const In*>(row0 + iw);
#pragma unroll
        for (int k = 0; k < 2 * NW; ++k) b[k] = __fadd_rn(o[k], b[k]);
      }
      __stcs(reinterpret_cast<In*>(row0 + iw), *reinterpret_cast<In*>(b));
    }
  }
}

// Backward of the 2x2 / stride 2 / no left-top padding case: every input element lies in
// exactly one window, so a thread takes one window pair (two horizontally adjacent outputs),
// finds the first tap (row-major) equal to the pooled value and adds dO there; avg spreads
// dO / count.  Same results as the gather form below, one pass, 128-bit accesses.
template <int MODE>
__global__ void __launch_bounds__(kThreads)
pool2x2_bwd_kernel(float* __restrict__ dI, const float* __restrict__ I, const float2* __restrict__ dO,
                   const float2* __restrict__ O, int64_t total2, int ih, int iw, int oh, int ow2, int acc) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < total2; gid += nthreads) {
    const int x2 = (int)(gid % ow2);
    const int64_t t = gid / ow2;
    const int y = (int)(t % oh);
    const int64_t plane = t / oh;
    const int64_t off0 = (plane * ih + 2 * y) * (int64_t)iw + 4 * x2;
    const bool has1 = (2 * y + 1) < ih;
    const float2 g = dO[gid];
    float4 ga = make_float4(0.f, 0.f, 0.f, 0.f), gb = ga;       // gradient of the two input rows
    if (MODE == LNN_POOL_AVG) {
      const float cnt = has1 ? 4.0f : 2.0f;
      const float q0 = __fdiv_rn(g.x, cnt), q1 = __fdiv_rn(g.y, cnt);
      ga = make_float4(q0, q0, q1, q1);
      gb = ga;
    } else {
      const float4 a = *reinterpret_cast<const float4*>(I + off0);
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (has1) b = *reinterpret_cast<const float4*>(I + off0 + iw);
      const float2 o = O[gid];
      // window 0: taps a.x, a.y, b.x, b.y in row-major order; window 1: a.z, a.w, b.z, b.w
      if (a.x == o.x) ga.x = g.x; else if (a.y == o.x) ga.y = g.x;
      else if (has1 && b.x == o.x) gb.x = g.x; else if (has1 && b.y == o.x) gb.y = g.x;
      if (a.z == o.y) ga.z = g.y; else if (a.w == o.y) ga.w = g.y;
      else if (has1 && b.z == o.y) gb.z = g.y; else if (has1 && b.w == o.y) gb.w = g.y;
    }
    float4* d0 = reinterpret_cast<float4*>(dI + off0);
    float4 v = acc ? *d0 : make_float4(0.f, 0.f, 0.f, 0.f);
    // the reference adds 0.0 + dO to its accumulator first, then accumulator to dI
    v.x = __fadd_rn(v.x, __fadd_rn(0.0f, ga.x)); v.y = __fadd_rn(v.y, __fadd_rn(0.0f, ga.y));
    v.z = __fadd_rn(v.z, __fadd_rn(0.0f, ga.z)); v.w = __fadd_rn(v.w, __fadd_rn(0.0f, ga.w));
    *d0 = v;
    if (has1) {
      float4* d1 = reinterpret_cast<float4*>(dI + off0 + iw);
      float4 w = acc ? *d1 : make_float4(0.f, 0.f, 0.f, 0.f);
      w.x = __fadd_rn(w.x, __fadd_rn(0.0f, gb.x)); w.y = __fadd_rn(w.y, __fadd_rn(0.0f, gb.y));
      w.z = __fadd_rn(w.z, __fadd_rn(0.0f, gb.z)); w.w = __fadd_rn(w.w, __fadd_rn(0.0f, gb.w));
      *d1 = w;
    }
  }
}

// Generic backward: one thread per INPUT element (so "+=" needs no atomics).  The windows that
// contain element (ih, iw) form a rectangle of outputs, oh in [oh_lo, oh_hi], ow likewise; their
// contributions are added from the highest (oh, ow) down, the order in which the reference meets
// them while it walks its taps upwards (pool2D.py:147-230), so overlapping windows accumulate
// identically.  avg: dO / (in-image size of the window).  max / min: dO if this element is the
// first one of the window, in row-major order, that equals the pooled value; the map of winners (idx)
// tells so without a second look at the window.
template <int MODE>
__global__ void __launch_bounds__(kThreads)
pool_bwd_kernel(float* __restrict__ dI, const float* __restrict__ I, const float* __restrict__ dO,
                const float* __restrict__ O, const uint8_t* __restrict__ idx, int64_t total, const PoolGeom g, int acc) {
  for (int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < total; gid += (int64_t)gridDim.x * blockDim.x) {
    int64_t pl;
    int ih, iw;
    split_index(gid, g.by_iw, g.by_ih, pl, ih, iw);
    const float* iplane = I ? I + pl * g.ih * g.iw : nullptr;
    const float* oplane = O ? O + pl * g.oh * g.ow : nullptr;
    const float* gplane = dO + pl * g.oh * g.ow;
    // windows covering the element: oh*stride - padt <= ih < oh*stride - padt + pool
    const int ah = ih + g.padt, aw = iw + g.padl;
    const int oh_hi = min((int)g.by_stride.div(ah), g.oh - 1), ow_hi = min((int)g.by_stride.div(aw), g.ow - 1);
    const int bh = ah - g.pool + g.stride, bw = aw - g.pool + g.stride;      // (a negative quotient counts as 0)
    const int oh_lo = bh > 0 ? (int)g.by_stride.div(bh) : 0, ow_lo = bw > 0 ? (int)g.by_stride.div(bw) : 0;
    float sum = 0.0f;
    for (int oh = oh_hi; oh >= oh_lo; --oh)
      for (int ow = ow_hi; ow >= ow_lo; --ow) {
        const float go = gplane[(int64_t)oh * g.ow + ow];
        if (MODE != LNN_POOL_AVG && idx) {
          const int place = (ah - oh * g.stride) * g.pool + aw - ow * g.stride;
          if (idx[(pl * g.oh + oh) * g.ow + ow] == place) sum = __fadd_rn(sum, go);
          continue;
        }
        const Window w = window_of(g, oh, ow);
        if (MODE == LNN_POOL_AVG) {
          sum = __fadd_rn(sum, __fdiv_rn(go, (float)((w.h1 - w.h0) * (w.w1 - w.w0))));
        } else {
          const float pooled = oplane[(int64_t)oh * g.ow + ow];
          if (iplane[(int64_t)ih * g.iw + iw] != pooled) continue;
          // is an earlier element of the window equal to the pooled value too?
          bool first = true;
          for (int h = w.h0; h <= ih && first; ++h) {
            const int stop = h == ih ? iw : w.w1;
            for (int x = w.w0; x < stop; ++x)
              if (iplane[(int64_t)h * g.iw + x] == pooled) { first = false; break; }
          }
          if (first) sum = __fadd_rn(sum, go);
        }
      }
    dI[gid] = __fadd_rn(acc ? dI[gid] : 0.0f, sum);
  }
}

inline int grid_for(const lnn::Device* d, int64_t work_items) {
  int64_t blocks = lnn_ceil_div(work_items, kThreads);
  int64_t cap = (int64_t)d->sm_count * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

// The window's place must fit the byte of a map of winners next to kNoWinner.
constexpr int kMaxIdxPool = 15;
// 2 or 1 windows per thread when the 2x2 kernels apply (big: the full-size tensor, small: the pooled one), else 0
inline int windows_per_thread(int ih, int iw, int oh, int ow, int pool, int stride, int padl, int padt, uint64_t big,
                              uint64_t small, uint64_t idx) {
  if (pool != 2 || stride != 2 || padl != 0 || padt != 0 || (iw & 1) || ow != iw / 2 || oh != (ih + 1) / 2) return 0;
  if ((iw & 3) == 0 && (big & 15) == 0 && (small & 7) == 0 && (idx & 1) == 0) return 2;
  return (big & 7) == 0 ? 1 : 0;
}

// Gradient of max_pool2D(2, 2) followed by the gradient of leaky_relu in one pass, WRITING dZ
// (the chain of the two un-fused gradient kernels reads and re-writes two zero-filled
// full-resolution tensors).  Y = leaky_relu(Z) is the pooled tensor's input, P its output, dP the
// gradient of P.  Per element exactly the roundings of the un-fused chain: the pooling gradient
// 0 + (0 + dP) at the first window position equal to P in row-major order (pool2D.py:147-230),
// then 0 + that * ((Y >= 0) + alpha * (Y < 0)) (element_wise_op.py:207-221; sign(Y) == sign(Z)).
__global__ void __launch_bounds__(kThreads)
pool2x2_lrelu_bwd_kernel(float* __restrict__ dZ, const float* __restrict__ Y, const float2* __restrict__ dP,
                         const float2* __restrict__ P, int64_t total2, int ih, int iw, int oh, int ow2,
                         float alpha, int act) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < total2; gid += nthreads) {
    const int x2 = (int)(gid % ow2);
    const int64_t t = gid / ow2;
    const int y = (int)(t % oh);
    const int64_t plane = t / oh;
    const int64_t off0 = (plane * ih + 2 * y) * (int64_t)iw + 4 * x2;
    const float4 a = __ldcs(reinterpret_cast<const float4*>(Y + off0));
    const float4 b = __ldcs(reinterpret_cast<const float4*>(Y + off0 + iw));
    const float2 g = dP[gid];
    const float2 o = P[gid];
    float ga[4] = {0.f, 0.f, 0.f, 0.f}, gb[4] = {0.f, 0.f, 0.f, 0.f};
    if (a.x == o.x) ga[0] = g.x; else if (a.y == o.x) ga[1] = g.x;
    else if (b.x == o.x) gb[0] = g.x; else if (b.y == o.x) gb[1] = g.x;
    if (a.z == o.y) ga[2] = g.y; else if (a.w == o.y) ga[3] = g.y;
    else if (b.z == o.y) gb[2] = g.y; else if (b.w == o.y) gb[3] = g.y;
    const float ya[4] = {a.x, a.y, a.z, a.w}, yb[4] = {b.x, b.y, b.z, b.w};
    float ra[4], rb[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float ua = __fadd_rn(0.0f, __fadd_rn(0.0f, ga[e]));
      float ub = __fadd_rn(0.0f, __fadd_rn(0.0f, gb[e]));
      if (act) {
        const float fa = __fadd_rn(ya[e] >= 0.0f ? 1.0f : 0.0f, __fmul_rn(alpha, ya[e] < 0.0f ? 1.0f : 0.0f));
        const float fb = __fadd_rn(yb[e] >= 0.0f ? 1.0f : 0.0f, __fmul_rn(alpha, yb[e] < 0.0f ? 1.0f : 0.0f));
        ua = __fadd_rn(0.0f, __fmul_rn(ua, fa));
        ub = __fadd_rn(0.0f, __fmul_rn(ub, fb));
      }
      ra[e] = ua; rb[e] = ub;
    }
    __stcs(reinterpret_cast<float4*>(dZ + off0), make_float4(ra[0], ra[1], ra[2], ra[3]));
    __stcs(reinterpret_cast<float4*>(dZ + off0 + iw), make_float4(rb[0], rb[1], rb[2], rb[3]));
  }
}

// The same gradient from the map of winning window positions a fused forward epilogue wrote
// (0..3 in row-major order, 4 = no position matched) instead of the full-resolution activation:
// the winner holds the pooled value itself, so leaky_relu' is taken from the sign of P, and every
// other position is +0 whatever its activation was.  T (optional, pooled size) receives the
// winner's value: its sum over (n, h, w) is the bias gradient.
__global__ void __launch_bounds__(kThreads)
pool2x2_idx_lrelu_bwd_kernel(float* __restrict__ dZ, float2* __restrict__ T, const uchar2* __restrict__ IDX,
                             const float2* __restrict__ dP, const float2* __restrict__ P, int64_t total2, int ih,
                             int iw, int oh, int ow2, float alpha, int act) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gid = tid; gid < total2; gid += nthreads) {
    const int x2 = (int)(gid % ow2);
    const int64_t t = gid / ow2;
    const int y = (int)(t % oh);
    const int64_t plane = t / oh;
    const int64_t off0 = (plane * ih + 2 * y) * (int64_t)iw + 4 * x2;
    const uchar2 w = IDX[gid];
    const float2 g = dP[gid];
    const float2 o = P[gid];
    float u[2] = {__fadd_rn(0.0f, __fadd_rn(0.0f, g.x)), __fadd_rn(0.0f, __fadd_rn(0.0f, g.y))};
    if (act) {
      const float f0 = __fadd_rn(o.x >= 0.0f ? 1.0f : 0.0f, __fmul_rn(alpha, o.x < 0.0f ? 1.0f : 0.0f));
      const float f1 = __fadd_rn(o.y >= 0.0f ? 1.0f : 0.0f, __fmul_rn(alpha, o.y < 0.0f ? 1.0f : 0.0f));
      u[0] = __fadd_rn(0.0f, __fmul_rn(u[0], f0));
      u[1] = __fadd_rn(0.0f, __fmul_rn(u[1], f1));
    }
    if (w.x > 3) u[0] = 0.0f;
    if (w.y > 3) u[1] = 0.0f;
    float ra[4] = {0.f, 0.f, 0.f, 0.f}, rb[4] = {0.f, 0.f, 0.f, 0.f};
    if (w.x == 0) ra[0] = u[0]; else if (w.x == 1) ra[1] = u[0]; else if (w.x == 2) rb[0] = u[0]; else if (w.x == 3) rb[1] = u[0];
    if (w.y == 0) ra[2] = u[1]; else if (w.y == 1) ra[3] = u[1]; else if (w.y == 2) rb[2] = u[1]; else if (w.y == 3) rb[3] = u[1];
    __stcs(reinterpret_cast<float4*>(dZ + off0), make_float4(ra[0], ra[1], ra[2], ra[3]));
    __stcs(reinterpret_cast<float4*>(dZ + off0 + iw), make_float4(rb[0], rb[1], rb[2], rb[3]));
    if (T) T[gid] = make_float2(u[0], u[1]);
  }
}

}  // namespace

extern "C" {

int lnn_pool2d_fwd(int dev, int mode, uint64_t O, uint64_t I, int64_t n, int64_t c, int ih, int iw,
                   int oh, int ow, int pool, int stride, int padl, int padt) {
  return lnn_pool2d_fwd_idx(dev, mode, O, 0, I, n, c, ih, iw, oh, ow, pool, stride, padl, padt);
}

int lnn_pool2d_fwd_idx(int dev, int mode, uint64_t O, uint64_t IDX, uint64_t I, int64_t n, int64_t c, int ih, int iw,
                       int oh, int ow, int pool, int stride, int padl, int padt) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(O && I, "null buffer");
  LNN_REQUIRE(n > 0 && c > 0 && ih > 0 && iw > 0 && oh > 0 && ow > 0, "bad extents");
  LNN_REQUIRE(pool >= 2 && stride >= 1, "pool_size must be >= 2 and stride >= 1");
  LNN_REQUIRE(mode >= 0 && mode <= 2, "unknown pool mode %d", mode);
  LNN_REQUIRE(!IDX || (mode != LNN_POOL_AVG && pool <= kMaxIdxPool), "no map of winners for this pooling");
  const int64_t total = n * c * oh * ow;
  float* o = (float*)(uintptr_t)O;
  uint8_t* idx = (uint8_t*)(uintptr_t)IDX;
  const float* i = (const float*)(uintptr_t)I;
  const int nw = windows_per_thread(ih, iw, oh, ow, pool, stride, padl, padt, I, O, IDX);
#define CALL(MODE)                                                                                                     \
  if (nw == 2 && idx)                                                                                                  \
    pool2x2_fwd_kernel<MODE, 2, MODE != LNN_POOL_AVG><<<grid_for(d, total / 2), kThreads, 0, d->stream>>>(             \
        o, idx, i, total / 2, ih, iw, lnn::FastDiv((uint32_t)ow / 2), lnn::FastDiv((uint32_t)oh));                     \
  else if (nw == 1 && idx)                                                                                             \
    pool2x2_fwd_kernel<MODE, 1, MODE != LNN_POOL_AVG><<<grid_for(d, total), kThreads, 0, d->stream>>>(                 \
        o, idx, i, total, ih, iw, lnn::FastDiv((uint32_t)ow), lnn::FastDiv((uint32_t)oh));                             \
  else if (nw == 2)                                                                                                    \
    pool2x2_fwd_kernel<MODE, 2, false><<<grid_for(d, total / 2), kThreads, 0, d->stream>>>(                                   \
        o, idx, i, total / 2, ih, iw, lnn::FastDiv((uint32_t)ow / 2), lnn::FastDiv((uint32_t)oh));                     \
  else if (nw == 1)                                                                                                    \
    pool2x2_fwd_kernel<MODE, 1, false><<<grid_for(d, total), kThreads, 0, d->stream>>>(                                \
        o, idx, i, total, ih, iw, lnn::FastDiv((uint32_t)ow), lnn::FastDiv((uint32_t)oh));                             \
  else                                                                                                                 \
    pool_fwd_kernel<MODE><<<grid_for(d, total), kThreads, 0, d->stream>>>(                                             \
        o, idx, i, total, PoolGeom(ih, iw, oh, ow, pool, stride, padl, padt))
  if (mode == LNN_POOL_AVG) { CALL(LNN_POOL_AVG); }
  else if (mode == LNN_POOL_MAX) { CALL(LNN_POOL_MAX); }
  else { CALL(LNN_POOL_MIN); }
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_pool2d_bwd_idx(int dev, int mode, uint64_t dI, uint64_t IDX, uint64_t dO, int64_t n, int64_t c, int ih, int iw,
                       int oh, int ow, int pool, int stride, int padl, int padt, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dI && dO, "null buffer");
  LNN_REQUIRE(mode >= 0 && mode <= 2, "unknown pool mode %d", mode);
  LNN_REQUIRE(n > 0 && c > 0 && ih > 0 && iw > 0 && oh > 0 && ow > 0, "bad extents");
  LNN_REQUIRE(pool >= 2 && stride >= 1, "pool_size must be >= 2 and stride >= 1");
  LNN_REQUIRE(mode == LNN_POOL_AVG || (IDX && pool <= kMaxIdxPool), "max / min need the map of winners");
  const int64_t total = n * c * oh * ow;
  float* di = (float*)(uintptr_t)dI;
  const uint8_t* idx = (const uint8_t*)(uintptr_t)IDX;
  const float* dout = (const float*)(uintptr_t)dO;
  const int nw = windows_per_thread(ih, iw, oh, ow, pool, stride, padl, padt, dI, dO, IDX);
#define CALL(MODE)                                                                                                     \
  if (nw == 2)                                                                                                         \
    pool2x2_bwd_idx_kernel<MODE, 2><<<grid_for(d, total / 2), kThreads, 0, d->stream>>>(                               \
        di, idx, dout, total / 2, ih, iw, lnn::FastDiv((uint32_t)ow / 2), lnn::FastDiv((uint32_t)oh), accumulate);     \
  else if (nw == 1)                                                                                                    \
    pool2x2_bwd_idx_kernel<MODE, 1><<<grid_for(d, total), kThreads, 0, d->stream>>>(                                   \
        di, idx, dout, total, ih, iw, lnn::FastDiv((uint32_t)ow), lnn::FastDiv((uint32_t)oh), accumulate);             \
  else                                                                                                                 \
    pool_bwd_kernel<MODE><<<grid_for(d, n * c * ih * iw), kThreads, 0, d->stream>>>(                                   \
        di, nullptr, dout, nullptr, idx, n * c * ih * iw, PoolGeom(ih, iw, oh, ow, pool, stride, padl, padt), accumulate)
  if (mode == LNN_POOL_AVG) { CALL(LNN_POOL_AVG); }
  else { CALL(LNN_POOL_MAX); }
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_pool2d_bwd(int dev, int mode, uint64_t dI, uint64_t I, uint64_t dO, uint64_t O, int64_t n,
                   int64_t c, int ih, int iw, int oh, int ow, int pool, int stride, int padl,
                   int padt) {
  return lnn_pool2d_bwd_acc(dev, mode, dI, I, dO, O, n, c, ih, iw, oh, ow, pool, stride, padl, padt, 1);
}

int lnn_pool2d_bwd_acc(int dev, int mode, uint64_t dI, uint64_t I, uint64_t dO, uint64_t O, int64_t n,
                       int64_t c, int ih, int iw, int oh, int ow, int pool, int stride, int padl,
                       int padt, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dI && dO, "null buffer");
  LNN_REQUIRE(mode >= 0 && mode <= 2, "unknown pool mode %d", mode);
  LNN_REQUIRE(mode == LNN_POOL_AVG || (I && O), "max/min backward needs I and O");
  LNN_REQUIRE(n > 0 && c > 0 && ih > 0 && iw > 0 && oh > 0 && ow > 0, "bad extents");
  LNN_REQUIRE(pool >= 2 && stride >= 1, "pool_size must be >= 2 and stride >= 1");
  const int64_t total = n * c * ih * iw;
  const PoolGeom g(ih, iw, oh, ow, pool, stride, padl, padt);
  float* di = (float*)(uintptr_t)dI;
  const float* i = (const float*)(uintptr_t)I;
  const float* dout = (const float*)(uintptr_t)dO;
  const float* o = (const float*)(uintptr_t)O;
  const bool fast = pool == 2 && stride == 2 && padl == 0 && padt == 0 && (iw % 4) == 0 &&
                    ow == iw / 2 && oh == (ih + 1) / 2 && (dI & 15) == 0 && (dO & 7) == 0 &&
                    (mode == LNN_POOL_AVG || ((I & 15) == 0 && (O & 7) == 0));
  if (fast) {
    const int64_t total2 = n * c * oh * (ow / 2);
    const int grid2 = grid_for(d, total2);
    if (mode == LNN_POOL_AVG)
      pool2x2_bwd_kernel<LNN_POOL_AVG><<<grid2, kThreads, 0, d->stream>>>(di, i, (const float2*)dout, (const float2*)o, total2, ih, iw, oh, ow / 2, accumulate);
    else if (mode == LNN_POOL_MAX)
      pool2x2_bwd_kernel<LNN_POOL_MAX><<<grid2, kThreads, 0, d->stream>>>(di, i, (const float2*)dout, (const float2*)o, total2, ih, iw, oh, ow / 2, accumulate);
    else
      pool2x2_bwd_kernel<LNN_POOL_MIN><<<grid2, kThreads, 0, d->stream>>>(di, i, (const float2*)dout, (const float2*)o, total2, ih, iw, oh, ow / 2, accumulate);
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  const int grid = grid_for(d, total);
  if (mode == LNN_POOL_AVG)
    pool_bwd_kernel<LNN_POOL_AVG><<<grid, kThreads, 0, d->stream>>>(di, i, dout, o, nullptr, total, g, accumulate);
  else if (mode == LNN_POOL_MAX)
    pool_bwd_kernel<LNN_POOL_MAX><<<grid, kThreads, 0, d->stream>>>(di, i, dout, o, nullptr, total, g, accumulate);
  else
    pool_bwd_kernel<LNN_POOL_MIN><<<grid, kThreads, 0, d->stream>>>(di, i, dout, o, nullptr, total, g, accumulate);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}


int lnn_pool2x2_idx_lrelu_bwd(int dev, uint64_t dZ, uint64_t T, uint64_t IDX, uint64_t P, uint64_t dP, int64_t n,
                              int64_t c, int ih, int iw, float alpha, int act) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dZ && IDX && P && dP, "null buffer");
  LNN_REQUIRE(n > 0 && c > 0 && ih > 0 && iw > 0, "bad extents");
  LNN_REQUIRE(act == 0 || act == 1, "unknown activation %d", act);
  if ((ih & 1) || (iw & 3) || (dZ & 15) || ((P | dP | T) & 7) || (IDX & 1))
    return lnn::set_error(LNN_E_UNSUPPORTED,
                          "fused pooling gradient needs an even height, a width that is a multiple of 4 and aligned buffers");
  const int oh = ih / 2, ow = iw / 2;
  const int64_t total2 = n * c * oh * (ow / 2);
  pool2x2_idx_lrelu_bwd_kernel<<<grid_for(d, total2), kThreads, 0, d->stream>>>(
      (float*)(uintptr_t)dZ, (float2*)(uintptr_t)T, (const uchar2*)(uintptr_t)IDX, (const float2*)(uintptr_t)dP,
      (const float2*)(uintptr_t)P, total2, ih, iw, oh, ow / 2, alpha, act);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_pool2x2_lrelu_bwd(int dev, uint64_t dZ, uint64_t Y, uint64_t P, uint64_t dP, int64_t n, int64_t c,
                          int ih, int iw, float alpha, int act) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dZ && Y && P && dP, "null buffer");
  LNN_REQUIRE(n > 0 && c > 0 && ih > 0 && iw > 0, "bad extents");
  LNN_REQUIRE(act == 0 || act == 1, "unknown activation %d", act);
  if ((ih & 1) || (iw & 3) || ((dZ | Y) & 15) || ((P | dP) & 7))
    return lnn::set_error(LNN_E_UNSUPPORTED,
                          "fused pooling gradient needs an even height, a width that is a multiple of 4 and aligned buffers");
  const int oh = ih / 2, ow = iw / 2;
  const int64_t total2 = n * c * oh * (ow / 2);
  pool2x2_lrelu_bwd_kernel<<<grid_for(d, total2), kThreads, 0, d->stream>>>(
      (float*)(uintptr_t)dZ, (const float*)(uintptr_t)Y, (const float2*)(uintptr_t)dP,
      (const float2*)(uintptr_t)P, total2, ih, iw, oh, ow / 2, alpha, act);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

}  // extern "C"
