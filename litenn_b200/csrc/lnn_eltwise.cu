// HBM-bound element-wise, broadcast-binary, fused scale+bias+leaky_relu, fill and SGD
// kernels.  Arithmetic follows the OpenCL C text the reference generates, with every
// literal single precision (the reference builds with -cl-single-precision-constant,
// litenn/core/minicl/CLDevice.py:93), comparisons converted int->float and multiplied
// in, and no fused multiply-add: each reference operator is its own rounding step, so
// the intrinsics __fmul_rn/__fadd_rn/__fsub_rn/__fdiv_rn are used throughout.
#include "lnn_common.cuh"
#include <algorithm>

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float b2f(bool c) { return c ? 1.0f : 0.0f; }

// ---- element-wise bodies (litenn/core/op/element_wise_op.py:112-364) -------------------

template <int OP>
__device__ __forceinline__ float ew_fwd(float I, float p0, float p1) {
  if (OP == LNN_EW_ABS) return fabsf(I);
  if (OP == LNN_EW_ADD_CONST) return fadd(I, p0);
  if (OP == LNN_EW_CLIP)
    return fadd(fadd(fmul(I, b2f((I >= p0) & (I <= p1))), fmul(p0, b2f(I < p0))),
                fmul(p1, b2f(I > p1)));
  if (OP == LNN_EW_COS) return cosf(I);
  if (OP == LNN_EW_EXP) return expf(I);
  if (OP == LNN_EW_LEAKY_RELU)
    return fadd(fmul(I, b2f(I >= 0.0f)), fmul(fmul(p0, I), b2f(I < 0.0f)));
  if (OP == LNN_EW_LOG) return logf(I);
  if (OP == LNN_EW_MUL_CONST) return fmul(I, p0);
  if (OP == LNN_EW_RDIV_CONST) return fdiv(p0, I);
  if (OP == LNN_EW_RSUB_CONST) return fsub(p0, I);
  if (OP == LNN_EW_RELU) return fmul(I, b2f(I >= 0.0f));
  if (OP == LNN_EW_SIGMOID) return fdiv(1.0f, fadd(1.0f, expf(-I)));
  if (OP == LNN_EW_SIN) return sinf(I);
  if (OP == LNN_EW_SQRT) return __fsqrt_rn(I);
  if (OP == LNN_EW_SQUARE) return fmul(I, I);
  if (OP == LNN_EW_TANH)
    return fsub(fdiv(2.0f, fadd(1.0f, expf(fmul(-2.0f, I)))), 1.0f);
  return 0.0f;
}

template <int OP>
__device__ __forceinline__ float ew_bwd(float I, float O, float dO, float p0, float p1, int flag) {
  if (OP == LNN_EW_ABS) return fmul(dO, fdiv(I, fabsf(I)));
  if (OP == LNN_EW_ADD_CONST) return dO;
  if (OP == LNN_EW_CLIP) return flag ? dO : fmul(dO, b2f((I >= p0) & (I <= p1)));
  if (OP == LNN_EW_COS) return fmul(dO, -sinf(I));
  if (OP == LNN_EW_EXP) return fmul(dO, expf(I));
  if (OP == LNN_EW_LEAKY_RELU)
    return fmul(dO, fadd(b2f(I >= 0.0f), fmul(p0, b2f(I < 0.0f))));
  if (OP == LNN_EW_LOG) return fmul(dO, fdiv(1.0f, I));
  if (OP == LNN_EW_MUL_CONST) return fmul(dO, p0);
  if (OP == LNN_EW_RDIV_CONST) return fmul(dO, -fdiv(p0, fmul(I, I)));
  if (OP == LNN_EW_RSUB_CONST) return -dO;
  if (OP == LNN_EW_RELU) return fmul(dO, b2f(I >= 0.0f));
  if (OP == LNN_EW_SIGMOID) return fmul(dO, fmul(O, fsub(1.0f, O)));
  if (OP == LNN_EW_SIN) return fmul(dO, cosf(I));
  if (OP == LNN_EW_SQRT) return fmul(dO, fdiv(1.0f, fmul(2.0f, __fsqrt_rn(I))));
  if (OP == LNN_EW_SQUARE) return fmul(fmul(dO, 2.0f), I);
  if (OP == LNN_EW_TANH) return fmul(dO, fsub(1.0f, fmul(O, O)));
  return 0.0f;
}

template <int OP>
__global__ void __launch_bounds__(kThreads)
ew_fwd_kernel(float* __restrict__ O, const float* __restrict__ I, int64_t n, float p0, float p1,
              int acc, int vec) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if (vec) {
    const int64_t n4 = n >> 2;
    const float4* I4 = reinterpret_cast<const float4*>(I);
    float4* O4 = reinterpret_cast<float4*>(O);
    for (int64_t i = tid; i < n4; i += nthreads) {
      float4 v = __ldcs(I4 + i);
      float4 r;
      r.x = ew_fwd<OP>(v.x, p0, p1); r.y = ew_fwd<OP>(v.y, p0, p1);
      r.z = ew_fwd<OP>(v.z, p0, p1); r.w = ew_fwd<OP>(v.w, p0, p1);
      if (acc) {
        float4 o = O4[i];
        r.x = fadd(o.x, r.x); r.y = fadd(o.y, r.y); r.z = fadd(o.z, r.z); r.w = fadd(o.w, r.w);
      }
      O4[i] = r;
    }
    for (int64_t i = (n4 << 2) + tid; i < n; i += nthreads) {
      float r = ew_fwd<OP>(I[i], p0, p1);
      O[i] = acc ? fadd(O[i], r) : r;
    }
  } else {
    for (int64_t i = tid; i < n; i += nthreads) {
      float r = ew_fwd<OP>(I[i], p0, p1);
      O[i] = acc ? fadd(O[i], r) : r;
    }
  }
}

// acc != 0: dI += ..., else dI = 0 + ... (a gradient nobody has touched yet: no zero fill, no read)
template <int OP>
__global__ void __launch_bounds__(kThreads)
ew_bwd_kernel(float* __restrict__ dI, const float* __restrict__ I, const float* __restrict__ O,
              const float* __restrict__ dO, int64_t n, float p0, float p1, int flag, int vec, int acc) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if (vec) {
    const int64_t n4 = n >> 2;
    for (int64_t i = tid; i < n4; i += nthreads) {
      float4 vi = reinterpret_cast<const float4*>(I)[i];
      float4 vo = reinterpret_cast<const float4*>(O)[i];
      float4 vd = reinterpret_cast<const float4*>(dO)[i];
      float4 g = acc ? reinterpret_cast<float4*>(dI)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      g.x = fadd(g.x, ew_bwd<OP>(vi.x, vo.x, vd.x, p0, p1, flag));
      g.y = fadd(g.y, ew_bwd<OP>(vi.y, vo.y, vd.y, p0, p1, flag));
      g.z = fadd(g.z, ew_bwd<OP>(vi.z, vo.z, vd.z, p0, p1, flag));
      g.w = fadd(g.w, ew_bwd<OP>(vi.w, vo.w, vd.w, p0, p1, flag));
      reinterpret_cast<float4*>(dI)[i] = g;
    }
    for (int64_t i = (n4 << 2) + tid; i < n; i += nthreads)
      dI[i] = fadd(acc ? dI[i] : 0.0f, ew_bwd<OP>(I[i], O[i], dO[i], p0, p1, flag));
  } else {
    for (int64_t i = tid; i < n; i += nthreads)
      dI[i] = fadd(acc ? dI[i] : 0.0f, ew_bwd<OP>(I[i], O[i], dO[i], p0, p1, flag));
  }
}

// ---- broadcast binary bodies (litenn/core/op/dual_wise_op.py:194-312) ------------------

template <int OP>
__device__ __forceinline__ float bin_fwd(float A, float B) {
  if (OP == LNN_BIN_ADD) return fadd(A, B);
  if (OP == LNN_BIN_SUB) return fsub(A, B);
  if (OP == LNN_BIN_MUL) return fmul(A, B);
  if (OP == LNN_BIN_DIV) return fdiv(A, B);
  if (OP == LNN_BIN_MAX) return fmaxf(A, B);
  if (OP == LNN_BIN_MIN) return fminf(A, B);
  if (OP == LNN_BIN_BCE)
    return fsub(fmul(-B, logf(A)), fmul(fsub(1.0f, B), logf(fsub(1.0f, A))));
  return 0.0f;
}

template <int OP, int WHICH>
__device__ __forceinline__ float bin_bwd(float A, float B, float O, float dO) {
  if (WHICH == 0) {
    if (OP == LNN_BIN_ADD || OP == LNN_BIN_SUB) return dO;
    if (OP == LNN_BIN_MUL) return fmul(dO, B);
    if (OP == LNN_BIN_DIV) return fdiv(dO, B);
    if (OP == LNN_BIN_MAX) return fmul(dO, b2f(A >= B));
    if (OP == LNN_BIN_MIN) return fmul(dO, b2f(A <= B));
    if (OP == LNN_BIN_BCE) return fdiv(fmul(dO, fsub(A, B)), fmul(A, fsub(1.0f, A)));
  } else {
    if (OP == LNN_BIN_ADD) return dO;
    if (OP == LNN_BIN_SUB) return -dO;
    if (OP == LNN_BIN_MUL) return fmul(dO, A);
    if (OP == LNN_BIN_DIV) return fmul(dO, -fdiv(A, fmul(B, B)));
    if (OP == LNN_BIN_MAX) return fmul(dO, b2f(A < B));
    if (OP == LNN_BIN_MIN) return fmul(dO, b2f(A > B));
    if (OP == LNN_BIN_BCE) return dO;
  }
  return 0.0f;
}

struct BcastDims {
  int rank;
  int64_t o[LNN_MAX_DIMS];     // output extents
  int64_t as[LNN_MAX_DIMS];    // element strides of A (0 where broadcast)
  int64_t bs[LNN_MAX_DIMS];
};

__device__ __forceinline__ void bcast_offsets(const BcastDims& d, int64_t gid, int64_t& ao,
                                              int64_t& bo) {
  ao = 0; bo = 0;
#pragma unroll
  for (int k = LNN_MAX_DIMS - 1; k >= 0; --k) {
    if (k < d.rank) {
      int64_t q = gid / d.o[k];
      int64_t r = gid - q * d.o[k];
      ao += r * d.as[k];
      bo += r * d.bs[k];
      gid = q;
    }
  }
}

// mode 0: forward; 1: dA; 2: dB.  same=1: no broadcasting at all (flat indexing).
template <int OP, int MODE>
__global__ void __launch_bounds__(kThreads)
bin_kernel(float* __restrict__ X, const float* __restrict__ A, const float* __restrict__ B,
           const float* __restrict__ O, const float* __restrict__ dO, int64_t n, BcastDims d,
           int acc, int same) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < n; i += nthreads) {
    int64_t ao = i, bo = i;
    if (!same) bcast_offsets(d, i, ao, bo);
    float a = A[ao], b = B[bo];
    float r;
    if (MODE == 0) {
      r = bin_fwd<OP>(a, b);
      X[i] = acc ? fadd(X[i], r) : r;
    } else {
      r = bin_bwd<OP, MODE - 1>(a, b, O[i], dO[i]);
      X[i] = fadd(acc ? X[i] : 0.0f, r);
    }
  }
}

// Fast broadcast path: every operand is the full tensor, one element, or varies along a
// single contiguous run of axes, so its element index is i, 0 or (i / inner) % size -- no
// per-axis index decomposition.  With vec != 0 a thread handles four consecutive outputs.
enum { OPM_FULL = 0, OPM_SCALAR = 1, OPM_AXIS = 2, OPM_GENERIC = 3 };
struct Operand { int mode; int64_t inner, size; };

__device__ __forceinline__ float op_load1(const float* __restrict__ p, const Operand& o, int64_t i) {
  if (o.mode == OPM_FULL) return p[i];
  if (o.mode == OPM_SCALAR) return __ldg(p);
  return __ldg(p + (i / o.inner) % o.size);
}
__device__ __forceinline__ float4 op_load4(const float* __restrict__ p, const Operand& o, int64_t i) {
  if (o.mode == OPM_FULL) return *reinterpret_cast<const float4*>(p + i);
  if (o.mode == OPM_SCALAR) { const float v = __ldg(p); return make_float4(v, v, v, v); }
  if (o.inner == 1) return __ldg(reinterpret_cast<const float4*>(p + i % o.size));
  const float v = __ldg(p + (i / o.inner) % o.size);
  return make_float4(v, v, v, v);
}

template <int OP, int MODE>
__global__ void __launch_bounds__(kThreads)
bin_fast_kernel(float* __restrict__ X, const float* __restrict__ A, const float* __restrict__ B,
                const float* __restrict__ O, const float* __restrict__ dO, int64_t n, Operand oa,
                Operand ob, int acc, int vec) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if (vec) {
    const int64_t n4 = n >> 2;
    for (int64_t q = tid; q < n4; q += nthreads) {
      const int64_t i = q << 2;
      const float4 a = op_load4(A, oa, i), b = op_load4(B, ob, i);
      float4 r;
      if (MODE == 0) {
        r.x = bin_fwd<OP>(a.x, b.x); r.y = bin_fwd<OP>(a.y, b.y);
        r.z = bin_fwd<OP>(a.z, b.z); r.w = bin_fwd<OP>(a.w, b.w);
      } else {
        const float4 o = *reinterpret_cast<const float4*>(O + i);
        const float4 g = *reinterpret_cast<const float4*>(dO + i);
        r.x = bin_bwd<OP, MODE - 1>(a.x, b.x, o.x, g.x); r.y = bin_bwd<OP, MODE - 1>(a.y, b.y, o.y, g.y);
        r.z = bin_bwd<OP, MODE - 1>(a.z, b.z, o.z, g.z); r.w = bin_bwd<OP, MODE - 1>(a.w, b.w, o.w, g.w);
      }
      float4* dst = reinterpret_cast<float4*>(X + i);
      if (acc || MODE != 0) {
        const float4 x = acc ? *dst : make_float4(0.f, 0.f, 0.f, 0.f);
        r.x = fadd(x.x, r.x); r.y = fadd(x.y, r.y); r.z = fadd(x.z, r.z); r.w = fadd(x.w, r.w);
      }
      *dst = r;
    }
    return;
  }
  for (int64_t i = tid; i < n; i += nthreads) {
    const float a = op_load1(A, oa, i), b = op_load1(B, ob, i);
    float r;
    if (MODE == 0) {
      r = bin_fwd<OP>(a, b);
      X[i] = acc ? fadd(X[i], r) : r;
    } else {
      r = bin_bwd<OP, MODE - 1>(a, b, O[i], dO[i]);
      X[i] = fadd(acc ? X[i] : 0.0f, r);
    }
  }
}

// y (+)= leaky_relu(x*g + b): x[N,C,HW]; each (n,c) plane is contiguous.  One float4 per
// thread per step; the channel index is recovered per vector (HW % 4 == 0 on this path).
__global__ void __launch_bounds__(kThreads)
scale_bias_lrelu_vec_kernel(float4* __restrict__ Y, const float4* __restrict__ X,
                            const float* __restrict__ G, const float* __restrict__ Bv,
                            int64_t n4, int64_t hw4, int64_t c, float alpha, int acc) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < n4; i += nthreads) {
    const int64_t ch = (i / hw4) % c;
    const float g = __ldg(G + ch), b = __ldg(Bv + ch);
    float4 v = __ldcs(X + i);
    float4 r;
    float t;
    t = fadd(fmul(v.x, g), b); r.x = fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f)));
    t = fadd(fmul(v.y, g), b); r.y = fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f)));
    t = fadd(fmul(v.z, g), b); r.z = fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f)));
    t = fadd(fmul(v.w, g), b); r.w = fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f)));
    if (acc) {
      float4 o = Y[i];
      r.x = fadd(o.x, r.x); r.y = fadd(o.y, r.y); r.z = fadd(o.z, r.z); r.w = fadd(o.w, r.w);
      Y[i] = r;
    } else {
      __stcs(Y + i, r);
    }
  }
}

__global__ void __launch_bounds__(kThreads)
scale_bias_lrelu_kernel(float* __restrict__ Y, const float* __restrict__ X,
                        const float* __restrict__ G, const float* __restrict__ Bv, int64_t n,
                        int64_t hw, int64_t c, float alpha, int acc) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < n; i += nthreads) {
    const int64_t ch = (i / hw) % c;
    float t = fadd(fmul(X[i], G[ch]), Bv[ch]);
    float r = fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f)));
    Y[i] = acc ? fadd(Y[i], r) : r;
  }
}

// Y = [leaky_relu](X [* G[c]] [+ B[c]]) for X viewed as [outer][channels][inner]: the reference's mul, add and
// leaky_relu kernels (dual_wise_op.py:194-204,283-295, element_wise_op.py:207-221) in one pass, each with
// its own rounding.  Null G / B and act = 0 leave a step out.  HBM-bound: one read, one write.
template <bool VEC>
__global__ void __launch_bounds__(kThreads)
channel_chain_fwd_kernel(float* __restrict__ Y, const float* __restrict__ X, const float* __restrict__ G,
                         const float* __restrict__ B, int64_t total, int64_t inner, int64_t channels, int act, float alpha) {
  constexpr int W = VEC ? 4 : 1;
  const int64_t step = (int64_t)gridDim.x * blockDim.x * W;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * W; i < total; i += step) {
    const int64_t ch = (i / inner) % channels;
    const float g = G ? __ldg(G + ch) : 1.0f, b = B ? __ldg(B + ch) : 0.0f;
    __align__(16) float v[W];
    if (VEC) *reinterpret_cast<float4*>(v) = __ldcs(reinterpret_cast<const float4*>(X + i));
    else v[0] = X[i];
#pragma unroll
    for (int e = 0; e < W; ++e) {
      float t = v[e];
      if (G) t = fmul(t, g);
      if (B) t = fadd(t, b);
      v[e] = act ? fadd(fmul(t, b2f(t >= 0.0f)), fmul(fmul(alpha, t), b2f(t < 0.0f))) : t;
    }
    if (VEC) __stcs(reinterpret_cast<float4*>(Y + i), *reinterpret_cast<float4*>(v));
    else Y[i] = v[0];
  }
}

// Gradients of that chain in one pass over X and dY: with t = X * G + B and dz = dY * leaky_relu'(t),
//   dX (+)= dz * G,   dG (+)= sum of dz * X,   dB (+)= sum of dz      (any of the three may be null).
// The reference runs four kernels with three full-size temporaries and two tree reductions.  S gives the
// sign of t when X, G or B have changed since the forward pass (the output, for alpha > 0); null: t is
// computed again.  A block owns one channel and a share of its elements, cut without regard to the outer
// axis, so that one image of few channels still covers the chip; its two sums meet the other blocks'
// through memory and the last one to arrive (a counter per channel) adds them in block order.  A thread
// adds up to thousands of terms in sequence, where the reference's tree adds pairs: beyond the four of a
// vector the sums are kept in 64 bits, which costs nothing next to the memory traffic.
template <bool VEC>
__global__ void __launch_bounds__(kThreads)
channel_chain_bwd_kernel(float* __restrict__ dX, float* __restrict__ dG, float* __restrict__ dB, const float* __restrict__ dY,
                         const float* __restrict__ X, const float* __restrict__ G, const float* __restrict__ B,
                         const float* __restrict__ S, int outer, int channels, int inner, int act, float alpha, int acc_x,
                         int acc_g, int acc_b, double2* __restrict__ partial, unsigned int* __restrict__ arrived) {
  constexpr int W = VEC ? 4 : 1;
  __shared__ double2 red[kThreads / 32];
  const int c = blockIdx.x, shares = gridDim.y, share = blockIdx.y;
  const float g = G ? __ldg(G + c) : 1.0f, b = B ? __ldg(B + c) : 0.0f;
  const uint32_t quads = (uint32_t)inner / W;            // vectors of one channel of one outer index
  const uint32_t work = (uint32_t)outer * quads, per = (work + shares - 1) / shares;
  const uint32_t e1 = min(work, ((uint32_t)share + 1) * per);     // shares * per < 2^31 + shares
  double sum_g = 0.0, sum_b = 0.0;
#pragma unroll 2
  for (uint32_t e = (uint32_t)share * per + threadIdx.x; e < e1; e += kThreads) {
    const uint32_t n = e / quads;
    const int64_t i = ((int64_t)n * channels + c) * inner + (int64_t)(e - n * quads) * W;
    float vec_g[W], vec_b[W];
    __align__(16) float x[W];
    __align__(16) float d[W];
    __align__(16) float s[W];
    if (VEC) {
      *reinterpret_cast<float4*>(x) = __ldcs(reinterpret_cast<const float4*>(X + i));
      *reinterpret_cast<float4*>(d) = __ldcs(reinterpret_cast<const float4*>(dY + i));
      if (S) *reinterpret_cast<float4*>(s) = __ldcs(reinterpret_cast<const float4*>(S + i));
    } else {
      x[0] = X[i]; d[0] = dY[i];
      if (S) s[0] = S[i];
    }
#pragma unroll
    for (int k = 0; k < W; ++k) {
      float dz = d[k];
      if (act) {
        float t = x[k];
        if (G) t = fmul(t, g);
        if (B) t = fadd(t, b);
        if (S) t = s[k];
        dz = fmul(dz, fadd(b2f(t >= 0.0f), fmul(alpha, b2f(t < 0.0f))));
      }
      vec_g[k] = fmul(dz, x[k]);
      vec_b[k] = dz;
      d[k] = G ? fmul(dz, g) : dz;
    }
    sum_g += VEC ? fadd(fadd(vec_g[0], vec_g[W > 1 ? 1 : 0]), fadd(vec_g[W > 2 ? 2 : 0], vec_g[W > 3 ? 3 : 0])) : vec_g[0];
    sum_b += VEC ? fadd(fadd(vec_b[0], vec_b[W > 1 ? 1 : 0]), fadd(vec_b[W > 2 ? 2 : 0], vec_b[W > 3 ? 3 : 0])) : vec_b[0];
    if (dX) {
      if (VEC) {
        float4* dst = reinterpret_cast<float4*>(dX + i);
        float4 o = acc_x ? *dst : make_float4(0.f, 0.f, 0.f, 0.f);
        o.x = fadd(o.x, d[0]); o.y = fadd(o.y, d[W > 1 ? 1 : 0]); o.z = fadd(o.z, d[W > 2 ? 2 : 0]); o.w = fadd(o.w, d[W > 3 ? 3 : 0]);
        __stcs(dst, o);
      } else {
        dX[i] = fadd(acc_x ? dX[i] : 0.0f, d[0]);
      }
    }
  }
  if (!dG && !dB) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum_g += __shfl_xor_sync(0xffffffffu, sum_g, o);
    sum_b += __shfl_xor_sync(0xffffffffu, sum_b, o);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_double2(sum_g, sum_b);
  __syncthreads();
  if (threadIdx.x >= 32) return;
  if (threadIdx.x == 0) {
    sum_g = red[0].x; sum_b = red[0].y;
    for (int w = 1; w < kThreads / 32; ++w) { sum_g += red[w].x; sum_b += red[w].y; }
  }
  if (shares > 1) {
    unsigned int before = 0u;
    if (threadIdx.x == 0) {
      __stcg(partial + (int64_t)c * shares + share, make_double2(sum_g, sum_b));
      __threadfence();
      before = atomicAdd(arrived + c, 1u);
      if (before == (unsigned)shares - 1) arrived[c] = 0u;
    }
    if (__shfl_sync(0xffffffffu, before, 0) != (unsigned)shares - 1) return;
    __threadfence();
    sum_g = sum_b = 0.0;
    for (int q = threadIdx.x; q < shares; q += 32) {
      const double2 v = __ldcg(partial + (int64_t)c * shares + q);
      sum_g += v.x; sum_b += v.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum_g += __shfl_xor_sync(0xffffffffu, sum_g, o);
      sum_b += __shfl_xor_sync(0xffffffffu, sum_b, o);
    }
  }
  if (threadIdx.x != 0) return;
  if (dG) dG[c] = fadd(acc_g ? dG[c] : 0.0f, (float)sum_g);
  if (dB) dB[c] = fadd(acc_b ? dB[c] : 0.0f, (float)sum_b);
}

__global__ void __launch_bounds__(kThreads)
fill_kernel(float* __restrict__ p, int64_t n, float v, int vec) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  if (vec) {
    const int64_t n4 = n >> 2;
    float4 v4 = make_float4(v, v, v, v);
    for (int64_t i = tid; i < n4; i += nthreads) reinterpret_cast<float4*>(p)[i] = v4;
    for (int64_t i = (n4 << 2) + tid; i < n; i += nthreads) p[i] = v;
  } else {
    for (int64_t i = tid; i < n; i += nthreads) p[i] = v;
  }
}

// A = -lr*G ; V += A  (litenn/core/optimizer/SGD.py:42-74 with momentum 0: the product
// is rounded, then added -- two kernels in the reference, two roundings here).
__global__ void __launch_bounds__(kThreads)
sgd_kernel(float* __restrict__ V, const float* __restrict__ G, int64_t n, float lr, float gscale,
           int use_scale) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < n; i += nthreads) {
    float g = G[i];
    if (use_scale) g = fmul(g, gscale);
    V[i] = fadd(V[i], fmul(-lr, g));
  }
}

inline int grid_for(const lnn::Device* d, int64_t work_items) {
  int64_t blocks = lnn_ceil_div(work_items, kThreads);
  int64_t cap = (int64_t)d->sm_count * 8;   // 8 resident blocks of 256 threads per SM
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

inline bool aligned16(uint64_t p) { return (p & 15) == 0; }

}  // namespace

#define EW_DISPATCH(OPV, CALL)                                                            \
  switch (OPV) {                                                                          \
    case LNN_EW_ABS: { CALL(LNN_EW_ABS); break; }                                         \
    case LNN_EW_ADD_CONST: { CALL(LNN_EW_ADD_CONST); break; }                             \
    case LNN_EW_CLIP: { CALL(LNN_EW_CLIP); break; }                                       \
    case LNN_EW_COS: { CALL(LNN_EW_COS); break; }                                         \
    case LNN_EW_EXP: { CALL(LNN_EW_EXP); break; }                                         \
    case LNN_EW_LEAKY_RELU: { CALL(LNN_EW_LEAKY_RELU); break; }                           \
    case LNN_EW_LOG: { CALL(LNN_EW_LOG); break; }                                         \
    case LNN_EW_MUL_CONST: { CALL(LNN_EW_MUL_CONST); break; }                             \
    case LNN_EW_RDIV_CONST: { CALL(LNN_EW_RDIV_CONST); break; }                           \
    case LNN_EW_RSUB_CONST: { CALL(LNN_EW_RSUB_CONST); break; }                           \
    case LNN_EW_RELU: { CALL(LNN_EW_RELU); break; }                                       \
    case LNN_EW_SIGMOID: { CALL(LNN_EW_SIGMOID); break; }                                 \
    case LNN_EW_SIN: { CALL(LNN_EW_SIN); break; }                                         \
    case LNN_EW_SQRT: { CALL(LNN_EW_SQRT); break; }                                       \
    case LNN_EW_SQUARE: { CALL(LNN_EW_SQUARE); break; }                                   \
    case LNN_EW_TANH: { CALL(LNN_EW_TANH); break; }                                       \
    default: return lnn::set_error(LNN_E_INVALID, "unknown element-wise op %d", OPV);     \
  }

#define BIN_DISPATCH(OPV, CALL)                                                           \
  switch (OPV) {                                                                          \
    case LNN_BIN_ADD: { CALL(LNN_BIN_ADD); break; }                                       \
    case LNN_BIN_SUB: { CALL(LNN_BIN_SUB); break; }                                       \
    case LNN_BIN_MUL: { CALL(LNN_BIN_MUL); break; }                                       \
    case LNN_BIN_DIV: { CALL(LNN_BIN_DIV); break; }                                       \
    case LNN_BIN_MAX: { CALL(LNN_BIN_MAX); break; }                                       \
    case LNN_BIN_MIN: { CALL(LNN_BIN_MIN); break; }                                       \
    case LNN_BIN_BCE: { CALL(LNN_BIN_BCE); break; }                                       \
    default: return lnn::set_error(LNN_E_INVALID, "unknown binary op %d", OPV);           \
  }

static int make_bcast(BcastDims& bd, int rank, const int64_t* o_shape, const int64_t* a_shape,
                      const int64_t* b_shape, int64_t* n_out, int* same) {
  LNN_REQUIRE(rank >= 1 && rank <= LNN_MAX_DIMS, "rank %d out of range", rank);
  LNN_REQUIRE(o_shape && a_shape && b_shape, "null shape");
  bd.rank = rank;
  int64_t n = 1, astr = 1, bstr = 1;
  *same = 1;
  for (int k = rank - 1; k >= 0; --k) {
    LNN_REQUIRE(o_shape[k] >= 1, "bad extent");
    LNN_REQUIRE(a_shape[k] == o_shape[k] || a_shape[k] == 1, "A axis %d not broadcastable", k);
    LNN_REQUIRE(b_shape[k] == o_shape[k] || b_shape[k] == 1, "B axis %d not broadcastable", k);
    bd.o[k] = o_shape[k];
    bd.as[k] = (a_shape[k] == 1) ? 0 : astr;
    bd.bs[k] = (b_shape[k] == 1) ? 0 : bstr;
    if (a_shape[k] != o_shape[k] || b_shape[k] != o_shape[k]) *same = 0;
    astr *= a_shape[k];
    bstr *= b_shape[k];
    n *= o_shape[k];
  }
  for (int k = rank; k < LNN_MAX_DIMS; ++k) { bd.o[k] = 1; bd.as[k] = 0; bd.bs[k] = 0; }
  *n_out = n;
  return LNN_OK;
}

// Classify one operand of a broadcast: FULL (same shape as the output), SCALAR (one element)
// or AXIS (its non-broadcast axes are one contiguous run: element = (i / inner) % size).
static void classify_operand(int rank, const int64_t* o_shape, const int64_t* x_shape, Operand& op) {
  int64_t x_size = 1, o_size = 1;
  for (int k = 0; k < rank; ++k) { x_size *= x_shape[k]; o_size *= o_shape[k]; }
  op.inner = 1; op.size = 1;
  if (x_size == o_size) { op.mode = OPM_FULL; return; }
  if (x_size == 1) { op.mode = OPM_SCALAR; return; }
  // find the run of axes where the operand is not broadcast (ignoring size-1 output axes)
  int first = -1, last = -1;
  for (int k = 0; k < rank; ++k)
    if (x_shape[k] != 1) { if (first < 0) first = k; last = k; }
  for (int k = first; k <= last; ++k)
    if (x_shape[k] != o_shape[k]) { op.mode = OPM_GENERIC; return; }
  for (int k = first; k <= last; ++k) op.size *= o_shape[k];
  for (int k = last + 1; k < rank; ++k) op.inner *= o_shape[k];
  op.mode = OPM_AXIS;
}

static bool operand_vec_ok(const Operand& op, uint64_t ptr) {
  if (op.mode == OPM_FULL) return (ptr & 15) == 0;
  if (op.mode == OPM_SCALAR) return true;
  if (op.mode == OPM_AXIS) return (op.inner % 4 == 0) || (op.inner == 1 && op.size % 4 == 0 && (ptr & 15) == 0);
  return false;
}

namespace {

__device__ __forceinline__ uint32_t pcg_hash(uint32_t v);

// ---- softmax and categorical cross-entropy over the rows of a [rows, cols] matrix -------------
// The reference composes them from exp, reduce_sum, div (softmax, element_wise_op.py:309-314) and
// clip, log, mul_const, mul, reduce_sum (categorical_crossentropy, dual_wise_op.py:228-250), nine
// launches and as many gradient launches.  Here one block owns a row: same operations in the
// same order per element (no max-subtraction, clip to [1e-7, 1 - 1e-7]) and the row sums in the
// reference's ceil-halving tree order (reduce.py:285-291), so forward values are identical.
constexpr int kRowThreads = 256;
constexpr int kRowMax = 8192;        // columns a block keeps in shared memory (32 KB)

// In-place ceil-halving tree over v[0..n): v[i] += v[i + ceil(n/2)], n = ceil(n/2), ... ; result in v[0].
__device__ __forceinline__ float row_tree_sum(float* v, int n) {
  while (n > 1) {
    const int h = (n + 1) >> 1;
    __syncthreads();
    for (int i = threadIdx.x; i + h < n; i += blockDim.x) v[i] = fadd(v[i], v[i + h]);
    n = h;
  }
  __syncthreads();
  return v[0];
}

__global__ void __launch_bounds__(kRowThreads)
softmax_fwd_kernel(float* __restrict__ P, const float* __restrict__ X, int64_t rows, int cols) {
  __shared__ float e[kRowMax];
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const float* x = X + r * cols;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) e[i] = expf(x[i]);
    const float s = row_tree_sum(e, cols);
    __syncthreads();
    // the tree consumed e: the quotient uses a fresh exp of the same input (same value)
    for (int i = threadIdx.x; i < cols; i += blockDim.x) P[r * cols + i] = fdiv(expf(x[i]), s);
    __syncthreads();
  }
}

// dX += (dP / s - sum_j(dP_j * e_j / s^2)) * e : the gradients of div (both operands), of the
// keepdims sum and of exp, in that association (dual_wise_op.py:268-281, reduce.py:250-260,
// element_wise_op.py:181-188)
__global__ void __launch_bounds__(kRowThreads)
softmax_bwd_kernel(float* __restrict__ dX, const float* __restrict__ X, const float* __restrict__ dP,
                   int64_t rows, int cols, int acc) {
  __shared__ float e[kRowMax];
  __shared__ float s_sh;
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const float* x = X + r * cols;
    const float* dp = dP + r * cols;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) e[i] = expf(x[i]);
    const float s = row_tree_sum(e, cols);
    __syncthreads();
    if (threadIdx.x == 0) s_sh = s;
    // ds = sum_j dP_j * (-e_j / (s * s))
    const float ss = fmul(s, s);
    for (int i = threadIdx.x; i < cols; i += blockDim.x) e[i] = fmul(dp[i], fdiv(-expf(x[i]), ss));
    const float ds = row_tree_sum(e, cols);
    __syncthreads();
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
      const float de = fadd(fdiv(dp[i], s), ds);
      dX[r * cols + i] = fadd(acc ? dX[r * cols + i] : 0.0f, fmul(de, expf(x[i])));
    }
    __syncthreads();
  }
}

// L[r] = sum_j (-T[r][j]) * log(clip(P[r][j], 1e-7, 1 - 1e-7)); T is [rows, cols] or one row (stride 0)
__global__ void __launch_bounds__(kRowThreads)
cce_fwd_kernel(float* __restrict__ L, const float* __restrict__ P, const float* __restrict__ T, int64_t rows,
               int cols, int64_t t_row_stride) {
  __shared__ float v[kRowMax];
  const float lo = 1e-7f, hi = fsub(1.0f, 1e-7f);
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const float* p = P + r * cols;
    const float* t = T + r * t_row_stride;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
      const float c = fminf(fmaxf(p[i], lo), hi);
      v[i] = fmul(fmul(t[i], -1.0f), logf(c));
    }
    const float s = row_tree_sum(v, cols);
    if (threadIdx.x == 0) L[r] = s;
    __syncthreads();
  }
}

// dP += dL[r] * (-T) * (1 / c) where the clip passed the value through (element_wise_op.py:133-139)
__global__ void __launch_bounds__(kThreads)
cce_bwd_kernel(float* __restrict__ dP, const float* __restrict__ P, const float* __restrict__ T,
               const float* __restrict__ dL, int64_t total, int64_t cols, int64_t t_row_stride, int acc) {
  const float lo = 1e-7f, hi = fsub(1.0f, 1e-7f);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / cols, j = i - r * cols;
    const float p = P[i];
    const float c = fminf(fmaxf(p, lo), hi);
    // reduce_sum' broadcasts dL; mul' gives dL * (-T); log' gives * (1 / c); clip' passes inside [lo, hi]
    const float dlog = fmul(dL[r], fmul(T[r * t_row_stride + j], -1.0f));
    const float dc = fmul(dlog, fdiv(1.0f, c));
    dP[i] = fadd(acc ? dP[i] : 0.0f, fmul(dc, (p >= lo && p <= hi) ? 1.0f : 0.0f));
  }
}

// One optimizer update per element, the reference's two or three kernels per tensor in one pass
// with the same operations in the same order (litenn/core/optimizer/SGD.py:42-83,
// RMSprop.py:37-69, Adam.py:43-84) and its learning-rate prologue (Optimizer.py:186-203):
// decay by 1 / (1 + lr_decay * iteration), then dropout of the step where the hash of
// (element index + seed) is <= lr_dropout.  SGD evaluates that prologue in both of its kernels,
// each with its own seed.  g is G * gscale when gscale != 1 (gradient averaging over replicas).
//
// One launch updates up to kOptTensors tensors (a launch per tensor cost a small network's step more
// than its forward pass): the blocks are dealt out to the tensors in chunks of kOptChunk elements.
constexpr int kOptTensors = 32;
constexpr int kOptChunk = 4 * kThreads;
struct OptTable {
  float* v[kOptTensors];
  const float* g[kOptTensors];
  float* s1[kOptTensors];
  float* s2[kOptTensors];
  int64_t n[kOptTensors];
  int64_t first[kOptTensors + 1];          // first chunk of each tensor
  uint32_t seed_a[kOptTensors], seed_b[kOptTensors];
  int count;
};

template <int KIND>
__device__ __forceinline__ void opt_element(float& v, float g, float& s1, float& s2, uint32_t i, float lr0,
                                            uint32_t seed_a, uint32_t seed_b, const lnn_opt_params& p) {
  const float uif = 1.0f / 4294967296.0f;
  if (p.gscale != 1.0f) g = fmul(g, p.gscale);
  float lr_a = lr0, lr_b = lr0;
  if (p.lr_dropout != 0.0f) {
    if (fmul(__uint2float_rn(pcg_hash(i + seed_a)), uif) <= p.lr_dropout) lr_a = 0.0f;
    if (fmul(__uint2float_rn(pcg_hash(i + seed_b)), uif) <= p.lr_dropout) lr_b = 0.0f;
  }
  if (KIND == LNN_OPT_SGD) {
    // A = momentum*A - lr*G ; V += A   (nesterov: V += momentum*A - lr*G with the new A)
    const float a = fsub(fmul(p.beta1, s1), fmul(lr_a, g));
    s1 = a;
    v = fadd(v, p.nesterov ? fsub(fmul(p.beta1, a), fmul(lr_b, g)) : a);
  } else if (KIND == LNN_OPT_RMSPROP) {
    // A = rho*A + (1-rho)*g*g ; V += -lr*G / (sqrt(A) + 1e-7)
    const float a = fadd(fmul(p.beta1, s1), fmul(fmul(fsub(1.0f, p.beta1), g), g));
    s1 = a;
    v = fadd(v, fdiv(fmul(-lr_b, g), fadd(__fsqrt_rn(a), 1e-7f)));
  } else {
    // M = b1*M + (1-b1)*G ; U = b2*U + (1-b2)*g*g ; V += -lr*M / (sqrt(U) + 1e-7)
    const float m = fadd(fmul(p.beta1, s1), fmul(fsub(1.0f, p.beta1), g));
    const float u = fadd(fmul(p.beta2, s2), fmul(fmul(fsub(1.0f, p.beta2), g), g));
    s1 = m; s2 = u;
    v = fadd(v, fdiv(fmul(-lr_b, m), fadd(__fsqrt_rn(u), 1e-7f)));
  }
}

template <int KIND>
__global__ void __launch_bounds__(kThreads)
opt_kernel(const __grid_constant__ OptTable t, const lnn_opt_params p) {
  float lr0 = p.lr;
  if (p.lr_decay != 0.0f) lr0 = fmul(lr0, fdiv(1.0f, fadd(1.0f, fmul(p.lr_decay, __uint2float_rn(p.iteration)))));
  const int64_t chunks = t.first[t.count];
  for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    int k = 0;
    while (c >= t.first[k + 1]) ++k;
    const int64_t i = (c - t.first[k]) * kOptChunk + (int64_t)threadIdx.x * 4;
    const int64_t n = t.n[k];
    if (i >= n) continue;
    float* v = t.v[k] + i;
    const float* g = t.g[k] + i;
    float* s1 = t.s1[k] + i;
    float* s2 = KIND == LNN_OPT_ADAM ? t.s2[k] + i : s1;
    const bool vec = i + 4 <= n && ((((uintptr_t)v | (uintptr_t)g | (uintptr_t)s1 | (uintptr_t)s2) & 15) == 0);
    if (vec) {
      float4 vv = *reinterpret_cast<float4*>(v), a = *reinterpret_cast<float4*>(s1), b = a;
      const float4 gg = *reinterpret_cast<const float4*>(g);
      if (KIND == LNN_OPT_ADAM) b = *reinterpret_cast<float4*>(s2);
      opt_element<KIND>(vv.x, gg.x, a.x, b.x, (uint32_t)i, lr0, t.seed_a[k], t.seed_b[k], p);
      opt_element<KIND>(vv.y, gg.y, a.y, b.y, (uint32_t)(i + 1), lr0, t.seed_a[k], t.seed_b[k], p);
      opt_element<KIND>(vv.z, gg.z, a.z, b.z, (uint32_t)(i + 2), lr0, t.seed_a[k], t.seed_b[k], p);
      opt_element<KIND>(vv.w, gg.w, a.w, b.w, (uint32_t)(i + 3), lr0, t.seed_a[k], t.seed_b[k], p);
      *reinterpret_cast<float4*>(v) = vv;
      *reinterpret_cast<float4*>(s1) = a;
      if (KIND == LNN_OPT_ADAM) *reinterpret_cast<float4*>(s2) = b;
    } else {
      for (int e = 0; e < 4 && i + e < n; ++e) {
        float b = KIND == LNN_OPT_ADAM ? s2[e] : 0.0f;
        opt_element<KIND>(v[e], g[e], s1[e], b, (uint32_t)(i + e), lr0, t.seed_a[k], t.seed_b[k], p);
        if (KIND == LNN_OPT_ADAM) s2[e] = b;
      }
    }
  }
}

// Random initializers: counter-based, one hash of (element index + seed) per element, so the
// result does not depend on the launch geometry.  PCG output functions as the reference uses
// them (litenn/core/CLKernelHelper.py:210-233; initializer/RandomUniform.py:12-20,
// RandomNormal.py:10-24); 2^-32 is the reference's 1 / (float)0xffffffff in single precision.
__device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {
  const uint32_t state = v * 747796405u + 2891336453u;
  const uint32_t word = ((state >> ((state >> 28) + 4u)) ^ state) * 277803737u;
  return (word >> 22) ^ word;
}
__device__ __forceinline__ void pcg2d_hash(uint32_t& a, uint32_t& b) {
  a = a * 1664525u + 1013904223u; b = b * 1664525u + 1013904223u;
  a += b * 1664525u; b += a * 1664525u;
  a ^= a >> 16; b ^= b >> 16;
  a += b * 1664525u; b += a * 1664525u;
  a ^= a >> 16; b ^= b >> 16;
}
constexpr float kUIF = 1.0f / 4294967296.0f;

__global__ void __launch_bounds__(kThreads)
init_uniform_kernel(float* __restrict__ O, int64_t n, uint32_t seed, float low, float high) {
  const float range = fsub(high, low);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float h = fmul(__uint2float_rn(pcg_hash((uint32_t)((uint64_t)i + seed))), kUIF);
    O[i] = fadd(fmul(h, range), low);
  }
}

__global__ void __launch_bounds__(kThreads)
init_normal_kernel(float* __restrict__ O, int64_t n, uint32_t seed, float mean, float stddev) {
  const float two_pi = 2.0f * 3.14159274101257f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t a = (uint32_t)((uint64_t)i + seed), b = 1u;
    pcg2d_hash(a, b);
    const float rx = fmul(__uint2float_rn(a), kUIF), ry = fmul(__uint2float_rn(b), kUIF);
    const float r = fmul(sqrtf(fmul(-2.0f, logf(rx))), cosf(fmul(two_pi, ry)));
    O[i] = fadd(mean, fmul(r, stddev));
  }
}

}  // namespace

extern "C" {

int lnn_init_uniform(int dev, uint64_t dst, int64_t count, uint32_t seed, float low, float high) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dst && count > 0, "bad arguments");
  init_uniform_kernel<<<grid_for(d, count), kThreads, 0, d->stream>>>((float*)(uintptr_t)dst, count, seed, low, high);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_init_normal(int dev, uint64_t dst, int64_t count, uint32_t seed, float mean, float stddev) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dst && count > 0, "bad arguments");
  init_normal_kernel<<<grid_for(d, count), kThreads, 0, d->stream>>>((float*)(uintptr_t)dst, count, seed, mean, stddev);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_fill_f32(int dev, uint64_t dst, int64_t count, float value) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dst && count > 0, "bad arguments");
  int vec = aligned16(dst);
  fill_kernel<<<grid_for(d, vec ? count / 4 + 1 : count), kThreads, 0, d->stream>>>(
      (float*)(uintptr_t)dst, count, value, vec);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_eltwise_fwd(int dev, int op, uint64_t O, uint64_t I, int64_t n, float p0, float p1,
                    int flag, int accumulate) {
  LNN_DEV(d, dev);
  (void)flag;
  LNN_REQUIRE(O && I && n > 0, "bad arguments");
  int vec = aligned16(O) && aligned16(I);
  int grid = grid_for(d, vec ? n / 4 + 1 : n);
#define CALL(OPC)                                                                         \
  ew_fwd_kernel<OPC><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)O,              \
      (const float*)(uintptr_t)I, n, p0, p1, accumulate, vec)
  EW_DISPATCH(op, CALL)
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_eltwise_bwd(int dev, int op, uint64_t dI, uint64_t I, uint64_t O, uint64_t dO, int64_t n,
                    float p0, float p1, int flag) {
  return lnn_eltwise_bwd_acc(dev, op, dI, I, O, dO, n, p0, p1, flag, 1);
}

int lnn_eltwise_bwd_acc(int dev, int op, uint64_t dI, uint64_t I, uint64_t O, uint64_t dO, int64_t n,
                        float p0, float p1, int flag, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dI && I && O && dO && n > 0, "bad arguments");
  int vec = aligned16(dI) && aligned16(I) && aligned16(O) && aligned16(dO);
  int grid = grid_for(d, vec ? n / 4 + 1 : n);
#define CALL(OPC)                                                                         \
  ew_bwd_kernel<OPC><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)dI,             \
      (const float*)(uintptr_t)I, (const float*)(uintptr_t)O, (const float*)(uintptr_t)dO, \
      n, p0, p1, flag, vec, accumulate)
  EW_DISPATCH(op, CALL)
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_binary_fwd(int dev, int op, uint64_t O, uint64_t A, uint64_t B, int rank,
                   const int64_t* o_shape, const int64_t* a_shape, const int64_t* b_shape,
                   int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(O && A && B, "null buffer");
  BcastDims bd; int64_t n; int same;
  int rc = make_bcast(bd, rank, o_shape, a_shape, b_shape, &n, &same);
  if (rc) return rc;
  Operand oa, ob;
  classify_operand(rank, o_shape, a_shape, oa);
  classify_operand(rank, o_shape, b_shape, ob);
  if (oa.mode != OPM_GENERIC && ob.mode != OPM_GENERIC) {
    const int vec = (n % 4 == 0) && aligned16(O) && operand_vec_ok(oa, A) && operand_vec_ok(ob, B);
    const int grid = grid_for(d, vec ? n / 4 : n);
#define CALL(OPC)                                                                         \
  bin_fast_kernel<OPC, 0><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)O,         \
      (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, nullptr, nullptr, n, oa, ob, \
      accumulate, vec)
    BIN_DISPATCH(op, CALL)
#undef CALL
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  int grid = grid_for(d, n);
#define CALL(OPC)                                                                         \
  bin_kernel<OPC, 0><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)O,              \
      (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, nullptr, nullptr, n, bd,    \
      accumulate, same)
  BIN_DISPATCH(op, CALL)
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_binary_bwd(int dev, int op, int which, uint64_t dX, uint64_t A, uint64_t B, uint64_t O,
                   uint64_t dO, int rank, const int64_t* o_shape, const int64_t* a_shape,
                   const int64_t* b_shape) {
  return lnn_binary_bwd_acc(dev, op, which, dX, A, B, O, dO, rank, o_shape, a_shape, b_shape, 1);
}

int lnn_binary_bwd_acc(int dev, int op, int which, uint64_t dX, uint64_t A, uint64_t B, uint64_t O,
                       uint64_t dO, int rank, const int64_t* o_shape, const int64_t* a_shape,
                       const int64_t* b_shape, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dX && A && B && O && dO, "null buffer");
  LNN_REQUIRE(which == 0 || which == 1, "which must be 0 or 1");
  BcastDims bd; int64_t n; int same;
  int rc = make_bcast(bd, rank, o_shape, a_shape, b_shape, &n, &same);
  if (rc) return rc;
  Operand oa, ob;
  classify_operand(rank, o_shape, a_shape, oa);
  classify_operand(rank, o_shape, b_shape, ob);
  if (oa.mode != OPM_GENERIC && ob.mode != OPM_GENERIC) {
    const int vec = (n % 4 == 0) && aligned16(dX) && aligned16(O) && aligned16(dO) &&
                    operand_vec_ok(oa, A) && operand_vec_ok(ob, B);
    const int grid = grid_for(d, vec ? n / 4 : n);
#define CALL(OPC)                                                                         \
  if (which == 0)                                                                         \
    bin_fast_kernel<OPC, 1><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)dX,      \
        (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, (const float*)(uintptr_t)O, \
        (const float*)(uintptr_t)dO, n, oa, ob, accumulate, vec);                                  \
  else                                                                                    \
    bin_fast_kernel<OPC, 2><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)dX,      \
        (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, (const float*)(uintptr_t)O, \
        (const float*)(uintptr_t)dO, n, oa, ob, accumulate, vec)
    BIN_DISPATCH(op, CALL)
#undef CALL
    LNN_CHECK_LAUNCH(d);
    return LNN_OK;
  }
  int grid = grid_for(d, n);
#define CALL(OPC)                                                                         \
  if (which == 0)                                                                         \
    bin_kernel<OPC, 1><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)dX,           \
        (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, (const float*)(uintptr_t)O, \
        (const float*)(uintptr_t)dO, n, bd, accumulate, same);                                     \
  else                                                                                    \
    bin_kernel<OPC, 2><<<grid, kThreads, 0, d->stream>>>((float*)(uintptr_t)dX,           \
        (const float*)(uintptr_t)A, (const float*)(uintptr_t)B, (const float*)(uintptr_t)O, \
        (const float*)(uintptr_t)dO, n, bd, accumulate, same)
  BIN_DISPATCH(op, CALL)
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_scale_bias_lrelu(int dev, uint64_t y, uint64_t x, uint64_t g, uint64_t b, int64_t n,
                         int64_t c, int64_t hw, float alpha, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(y && x && g && b && n > 0 && c > 0 && hw > 0, "bad arguments");
  int64_t total = n * c * hw;
  if ((hw & 3) == 0 && aligned16(y) && aligned16(x)) {
    int64_t n4 = total >> 2;
    scale_bias_lrelu_vec_kernel<<<grid_for(d, n4), kThreads, 0, d->stream>>>(
        (float4*)(uintptr_t)y, (const float4*)(uintptr_t)x, (const float*)(uintptr_t)g,
        (const float*)(uintptr_t)b, n4, hw >> 2, c, alpha, accumulate);
  } else {
    scale_bias_lrelu_kernel<<<grid_for(d, total), kThreads, 0, d->stream>>>(
        (float*)(uintptr_t)y, (const float*)(uintptr_t)x, (const float*)(uintptr_t)g,
        (const float*)(uintptr_t)b, total, hw, c, alpha, accumulate);
  }
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_channel_chain_fwd(int dev, uint64_t Y, uint64_t X, uint64_t G, uint64_t B, int64_t outer, int64_t channels,
                          int64_t inner, int act, float alpha) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(Y && X && outer > 0 && channels > 0 && inner > 0, "bad arguments");
  const int64_t total = outer * channels * inner;
  if ((inner & 3) == 0 && aligned16(Y) && aligned16(X))
    channel_chain_fwd_kernel<true><<<grid_for(d, total / 4), kThreads, 0, d->stream>>>(
        (float*)(uintptr_t)Y, (const float*)(uintptr_t)X, (const float*)(uintptr_t)G, (const float*)(uintptr_t)B, total, inner,
        channels, act, alpha);
  else
    channel_chain_fwd_kernel<false><<<grid_for(d, total), kThreads, 0, d->stream>>>(
        (float*)(uintptr_t)Y, (const float*)(uintptr_t)X, (const float*)(uintptr_t)G, (const float*)(uintptr_t)B, total, inner,
        channels, act, alpha);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_channel_chain_bwd(int dev, uint64_t dX, uint64_t dG, uint64_t dB, uint64_t dY, uint64_t X, uint64_t G, uint64_t B,
                          uint64_t S, int64_t outer, int64_t channels, int64_t inner, int act, float alpha, int acc_x,
                          int acc_g, int acc_b) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dY && X && outer > 0 && channels > 0 && inner > 0, "bad arguments");
  // (the host layer puts a chain off under the same limits: a channel's elements are counted in 32 bits)
  LNN_REQUIRE(outer < (1ll << 31) && channels < (1ll << 30) && inner < (1ll << 31) && outer * inner < (1ll << 31),
              "extents too large for the fused gradient");
  // as many blocks as are resident at once (eight per SM), but at least two vectors per thread of each
  const bool vec = (inner & 3) == 0 && aligned16(X | dY | S | dX);
  const int64_t vectors = outer * (inner / (vec ? 4 : 1));
  int64_t shares = std::min<int64_t>((int64_t)d->sm_count * 8 / channels, vectors / (2 * kThreads));
  shares = channels > lnn::kTileCounters ? 1 : std::max<int64_t>(1, shares);
  lnn::Scratch part(d);
  if (shares > 1 && (dG || dB)) {
    const int rc = part.get((uint64_t)shares * channels * sizeof(double2));
    if (rc) return rc;
  }
  const dim3 grid((unsigned)channels, (unsigned)shares);
#define CALL(VEC)                                                                                                  \
  channel_chain_bwd_kernel<VEC><<<grid, kThreads, 0, d->stream>>>(                                                 \
      (float*)(uintptr_t)dX, (float*)(uintptr_t)dG, (float*)(uintptr_t)dB, (const float*)(uintptr_t)dY,            \
      (const float*)(uintptr_t)X, (const float*)(uintptr_t)G, (const float*)(uintptr_t)B, (const float*)(uintptr_t)S, \
      (int)outer, (int)channels, (int)inner, act, alpha, acc_x, acc_g, acc_b, part.as<double2>(), d->tile_counters)
  if (vec) CALL(true);
  else CALL(false);
#undef CALL
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_softmax_fwd(int dev, uint64_t P, uint64_t X, int64_t rows, int64_t cols) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(P && X && rows > 0 && cols > 0, "bad arguments");
  LNN_REQUIRE(cols <= kRowMax, "rows longer than %d elements are not supported by the fused softmax", kRowMax);
  softmax_fwd_kernel<<<(unsigned)std::min<int64_t>(rows, (int64_t)d->sm_count * 8), kRowThreads, 0, d->stream>>>(
      (float*)(uintptr_t)P, (const float*)(uintptr_t)X, rows, (int)cols);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_softmax_bwd(int dev, uint64_t dX, uint64_t X, uint64_t dP, int64_t rows, int64_t cols) {
  return lnn_softmax_bwd_acc(dev, dX, X, dP, rows, cols, 1);
}

int lnn_softmax_bwd_acc(int dev, uint64_t dX, uint64_t X, uint64_t dP, int64_t rows, int64_t cols, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dX && X && dP && rows > 0 && cols > 0 && cols <= kRowMax, "bad arguments");
  softmax_bwd_kernel<<<(unsigned)std::min<int64_t>(rows, (int64_t)d->sm_count * 8), kRowThreads, 0, d->stream>>>(
      (float*)(uintptr_t)dX, (const float*)(uintptr_t)X, (const float*)(uintptr_t)dP, rows, (int)cols, accumulate);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_cce_fwd(int dev, uint64_t L, uint64_t P, uint64_t T, int64_t rows, int64_t cols, int64_t t_row_stride) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(L && P && T && rows > 0 && cols > 0 && cols <= kRowMax, "bad arguments");
  cce_fwd_kernel<<<(unsigned)std::min<int64_t>(rows, (int64_t)d->sm_count * 8), kRowThreads, 0, d->stream>>>(
      (float*)(uintptr_t)L, (const float*)(uintptr_t)P, (const float*)(uintptr_t)T, rows, (int)cols, t_row_stride);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_cce_bwd(int dev, uint64_t dP, uint64_t P, uint64_t T, uint64_t dL, int64_t rows, int64_t cols,
                int64_t t_row_stride) {
  return lnn_cce_bwd_acc(dev, dP, P, T, dL, rows, cols, t_row_stride, 1);
}

int lnn_cce_bwd_acc(int dev, uint64_t dP, uint64_t P, uint64_t T, uint64_t dL, int64_t rows, int64_t cols,
                    int64_t t_row_stride, int accumulate) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(dP && P && T && dL && rows > 0 && cols > 0, "bad arguments");
  cce_bwd_kernel<<<grid_for(d, rows * cols), kThreads, 0, d->stream>>>(
      (float*)(uintptr_t)dP, (const float*)(uintptr_t)P, (const float*)(uintptr_t)T, (const float*)(uintptr_t)dL,
      rows * cols, cols, t_row_stride, accumulate);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

int lnn_optimizer_step(int dev, int kind, uint64_t V, uint64_t G, uint64_t S1, uint64_t S2, int64_t n,
                       const lnn_opt_params* p) {
  LNN_REQUIRE(p, "bad arguments");
  const uint32_t seeds[2] = {p->seed_a, p->seed_b};
  return lnn_optimizer_step_many(dev, kind, 1, &V, &G, &S1, S2 ? &S2 : nullptr, &n, seeds, p);
}

int lnn_optimizer_step_many(int dev, int kind, int count, const uint64_t* V, const uint64_t* G, const uint64_t* S1,
                            const uint64_t* S2, const int64_t* n, const uint32_t* seeds, const lnn_opt_params* p) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(count > 0 && V && G && n && p, "bad arguments");
  LNN_REQUIRE(kind >= LNN_OPT_SGD && kind <= LNN_OPT_ADAM, "unknown optimizer kind %d", kind);
  LNN_REQUIRE(S1 && (kind != LNN_OPT_ADAM || S2), "optimizer state buffer missing");
  for (int at = 0; at < count; at += kOptTensors) {
    OptTable t;
    t.count = std::min(count - at, kOptTensors);
    t.first[0] = 0;
    for (int k = 0; k < t.count; ++k) {
      const int j = at + k;
      LNN_REQUIRE(V[j] && G[j] && n[j] > 0, "bad arguments");
      LNN_REQUIRE(S1[j] && (kind != LNN_OPT_ADAM || S2[j]), "optimizer state buffer missing");
      t.v[k] = (float*)(uintptr_t)V[j]; t.g[k] = (const float*)(uintptr_t)G[j];
      t.s1[k] = (float*)(uintptr_t)S1[j]; t.s2[k] = S2 ? (float*)(uintptr_t)S2[j] : nullptr;
      t.n[k] = n[j];
      t.seed_a[k] = seeds ? seeds[2 * j] : 0u; t.seed_b[k] = seeds ? seeds[2 * j + 1] : 0u;
      t.first[k + 1] = t.first[k] + lnn_ceil_div(n[j], kOptChunk);
    }
    const unsigned grid = (unsigned)std::min<int64_t>(t.first[t.count], (int64_t)d->sm_count * 8);
    if (kind == LNN_OPT_SGD) opt_kernel<LNN_OPT_SGD><<<grid, kThreads, 0, d->stream>>>(t, *p);
    else if (kind == LNN_OPT_RMSPROP) opt_kernel<LNN_OPT_RMSPROP><<<grid, kThreads, 0, d->stream>>>(t, *p);
    else opt_kernel<LNN_OPT_ADAM><<<grid, kThreads, 0, d->stream>>>(t, *p);
    LNN_CHECK_LAUNCH(d);
  }
  return LNN_OK;
}

int lnn_sgd_step(int dev, uint64_t V, uint64_t G, int64_t n, float lr, float gscale) {
  LNN_DEV(d, dev);
  LNN_REQUIRE(V && G && n > 0, "bad arguments");
  sgd_kernel<<<grid_for(d, n), kThreads, 0, d->stream>>>(
      (float*)(uintptr_t)V, (const float*)(uintptr_t)G, n, lr, gscale, gscale != 1.0f);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

}  // extern "C"
