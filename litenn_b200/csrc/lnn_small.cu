// Matrix products too small for the tensor-core engine.
//
// The engine needs its operands scaled and split first (two launches per operand) and spends some
// ten microseconds on TMEM, barriers and the pipeline ramp of one 128 x N tile however little there
// is to multiply; below a few hundred MFLOP that is all the time there is.  Here one launch reads the
// fp32 operands as they are and multiplies on the FP32 pipe (exact products, fp32 sums).
//
// What bounds it is latency: global loads of one K slab, then the next.  So tiles are 32 x 32, the next
// slab is loaded into registers while the current one is multiplied, and K is cut twice: four groups of
// 64 threads of a block take a quarter each (partial sums meet in shared memory), and up to eight
// blocks of a cluster take a piece each (they meet through distributed shared memory).  Every sum is
// taken in a fixed order.  [64, 256] x [256, 512]: 31 us in five launches before, 5 us in one; partial
// sums through global memory with an arrival counter took 8 us.  Products with enough (and well filled) 64 x 64
// tiles to cover the SMs twice take those, whole K each: half the operand traffic per multiply-add.
#include "lnn_common.cuh"
#include <cooperative_groups.h>
#include <algorithm>

namespace {

struct SmallGemm {
  float* C;
  const float* A;
  const float* B;
  const float* bias;
  int64_t stride_a, stride_b, stride_c;      // between the matrices of a batch
  int m, n, k;
  int tiles_m, splits, k_per_split;          // splits = blocks of a cluster
  int accumulate;
  int vec_a, vec_b, vec_c;                   // 128-bit loads / stores are aligned and in range
};

// Four consecutive elements along the contiguous axis of an operand: `lim` of them exist.
__device__ __forceinline__ float4 load4(const float* p, int lim, int vec) {
  if (vec && lim >= 4) return __ldg(reinterpret_cast<const float4*>(p));
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (lim > 0) v.x = __ldg(p);
  if (lim > 1) v.y = __ldg(p + 1);
  if (lim > 2) v.z = __ldg(p + 2);
  if (lim > 3) v.w = __ldg(p + 3);
  return v;
}

// One operand tile of EXT (rows of C / columns of C) x BK in registers and from there to shared memory as
// S[k][ext].  KFAST: the operand is contiguous along K in memory ([ext][k]), else along ext ([k][ext]).
template <int EXT, int BK, int THREADS, bool KFAST>
struct Operand {
  static constexpr int kVecs = EXT * BK / 4 / THREADS;
  static_assert(kVecs * 4 * THREADS == EXT * BK, "the tile is a whole number of vectors per thread");
  static constexpr int kPitch = EXT + 4;
  float4 r[kVecs];
  __device__ __forceinline__ void load(int tid, const float* __restrict__ p, int64_t ld, int e0, int ext, int k0, int k_end, int vec) {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int v = tid + i * THREADS;
      if (KFAST) {
        const int e = e0 + v / (BK / 4), k = k0 + (v % (BK / 4)) * 4;
        r[i] = load4(p + (int64_t)e * ld + k, e < ext ? k_end - k : 0, vec);
      } else {
        const int k = k0 + v / (EXT / 4), e = e0 + (v % (EXT / 4)) * 4;
        r[i] = load4(p + (int64_t)k * ld + e, k < k_end ? ext - e : 0, vec);
      }
    }
  }
  __device__ __forceinline__ void store(int tid, float* S) const {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int v = tid + i * THREADS;
      if (KFAST) {
        const int e = v / (BK / 4), k = (v % (BK / 4)) * 4;
        S[(k + 0) * kPitch + e] = r[i].x; S[(k + 1) * kPitch + e] = r[i].y;
        S[(k + 2) * kPitch + e] = r[i].z; S[(k + 3) * kPitch + e] = r[i].w;
      } else {
        const int k = v / (EXT / 4), e = (v % (EXT / 4)) * 4;
        *reinterpret_cast<float4*>(S + k * kPitch + e) = r[i];
      }
    }
  }
};

// One row of four results of C.
__device__ __forceinline__ void write4(const SmallGemm& p, int batch, int m, int n, float4 v) {
  if (m >= p.m || n >= p.n) return;
  float* dst = p.C + batch * p.stride_c + (int64_t)m * p.n + n;
  float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (p.bias && n + j < p.n) e[j] = __fadd_rn(e[j], __ldg(p.bias + n + j));
  if (p.vec_c && n + 4 <= p.n) {
    float4 o = make_float4(e[0], e[1], e[2], e[3]);
    if (p.accumulate) {
      const float4 old = *reinterpret_cast<const float4*>(dst);
      o.x = __fadd_rn(old.x, o.x); o.y = __fadd_rn(old.y, o.y); o.z = __fadd_rn(old.z, o.z); o.w = __fadd_rn(old.w, o.w);
    }
    *reinterpret_cast<float4*>(dst) = o;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.n) dst[j] = p.accumulate ? __fadd_rn(dst[j], e[j]) : e[j];
  }
}

__device__ __forceinline__ void group_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// GROUPS groups of (EXT / 4)^2 threads, each with a 4 x 4 piece of the EXT x EXT tile per thread.
template <int EXT, int BK, int GROUPS, bool A_KFAST, bool B_KFAST>
__global__ void __launch_bounds__(GROUPS * (EXT / 4) * (EXT / 4))
small_gemm_kernel(const SmallGemm p) {
  constexpr int THREADS = (EXT / 4) * (EXT / 4), SIDE = EXT / 4;
  typedef Operand<EXT, BK, THREADS, A_KFAST> OpA;
  typedef Operand<EXT, BK, THREADS, B_KFAST> OpB;
  constexpr int kTile = BK * OpA::kPitch;
  __shared__ __align__(16) float sa[GROUPS][2][kTile];
  __shared__ __align__(16) float sb[GROUPS][2][kTile];
  static_assert(GROUPS == 1 || sizeof(sa) >= sizeof(float) * GROUPS * EXT * EXT, "partial sums reuse the operand tiles");
  const int group = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
  const int batch = blockIdx.z, split = blockIdx.y;
  const int m0 = (blockIdx.x % p.tiles_m) * EXT, n0 = (blockIdx.x / p.tiles_m) * EXT;
  const int per_group = (p.k_per_split / GROUPS + BK - 1) / BK * BK;
  const int split_end = min(p.k, (split + 1) * p.k_per_split);
  const int k_begin = split * p.k_per_split + group * per_group;
  const int k_end = GROUPS == 1 ? split_end : min(split_end, k_begin + per_group);
  const float* A = p.A + batch * p.stride_a;
  const float* B = p.B + batch * p.stride_b;
  const int64_t lda = A_KFAST ? p.k : p.m, ldb = B_KFAST ? p.k : p.n;
  const int tx = tid % SIDE, ty = tid / SIDE;
  OpA a;
  OpB b;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  a.load(tid, A, lda, m0, p.m, k_begin, k_end, p.vec_a);
  b.load(tid, B, ldb, n0, p.n, k_begin, k_end, p.vec_b);
  int buf = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += BK) {
    a.store(tid, sa[group][buf]);
    b.store(tid, sb[group][buf]);
    if (GROUPS == 1) __syncthreads();
    else group_barrier(1 + group, THREADS);
    if (k0 + BK < k_end) {
      a.load(tid, A, lda, m0, p.m, k0 + BK, k_end, p.vec_a);
      b.load(tid, B, ldb, n0, p.n, k0 + BK, k_end, p.vec_b);
    }
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 y = *reinterpret_cast<const float4*>(&sb[group][buf][k * OpB::kPitch + tx * 4]);
      const float4 q = *reinterpret_cast<const float4*>(&sa[group][buf][k * OpA::kPitch + ty * 4]);
      const float x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = __fmaf_rn(x[i], y.x, acc[i][0]); acc[i][1] = __fmaf_rn(x[i], y.y, acc[i][1]);
        acc[i][2] = __fmaf_rn(x[i], y.z, acc[i][2]); acc[i][3] = __fmaf_rn(x[i], y.w, acc[i][3]);
      }
    }
    buf ^= 1;                      // the other buffer was last read before the barrier just passed
  }
  if (GROUPS == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      write4(p, batch, m0 + ty * 4 + i, n0 + tx * 4, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
    return;
  }
  // groups: sums[group][row][col] in the memory of the operand tiles, one row of four per thread and step
  __syncthreads();
  float4* sums = reinterpret_cast<float4*>(&sa[0][0][0]);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    sums[(group * EXT + ty * 4 + i) * SIDE + tx] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  constexpr int kQuads = EXT * SIDE;                       // float4 values of a tile
  for (int q = threadIdx.x; q < kQuads; q += GROUPS * THREADS) {
    float4 v = sums[q];
#pragma unroll
    for (int g = 1; g < GROUPS; ++g) {
      const float4 o = sums[g * kQuads + q];
      v.x = __fadd_rn(v.x, o.x); v.y = __fadd_rn(v.y, o.y); v.z = __fadd_rn(v.z, o.z); v.w = __fadd_rn(v.w, o.w);
    }
    if (p.splits == 1) write4(p, batch, m0 + q / SIDE, n0 + (q % SIDE) * 4, v);
    else sums[q] = v;
  }
  if (p.splits == 1) return;
  // blocks of the cluster: each finishes its share of the tile's rows
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int q = split * (GROUPS * THREADS) + threadIdx.x; q < kQuads; q += p.splits * GROUPS * THREADS) {
    float4 v = cluster.map_shared_rank(sums, 0)[q];
    for (int r = 1; r < p.splits; ++r) {
      const float4 o = cluster.map_shared_rank(sums, r)[q];
      v.x = __fadd_rn(v.x, o.x); v.y = __fadd_rn(v.y, o.y); v.z = __fadd_rn(v.z, o.z); v.w = __fadd_rn(v.w, o.w);
    }
    write4(p, batch, m0 + q / SIDE, n0 + (q % SIDE) * 4, v);
  }
  cluster.sync();                  // nobody leaves while its shared memory is being read
}

template <int EXT, int BK, int GROUPS>
int launch(lnn::Device* d, SmallGemm& p, int batch, int trans_a, int trans_b) {
  p.tiles_m = (p.m + EXT - 1) / EXT;
  const int64_t tiles = (int64_t)p.tiles_m * ((p.n + EXT - 1) / EXT);
  p.splits = 1;
  if (GROUPS > 1)
    while (p.splits < 8 && tiles * batch * p.splits * 2 <= 2 * d->sm_count && p.k >= p.splits * 2 * GROUPS * BK) p.splits *= 2;
  p.k_per_split = (p.k + p.splits - 1) / p.splits;
  p.k_per_split = (p.k_per_split + GROUPS * BK - 1) / (GROUPS * BK) * (GROUPS * BK);   // (a block may be left without any)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)p.splits, (unsigned)batch);
  cfg.blockDim = dim3(GROUPS * (EXT / 4) * (EXT / 4));
  cfg.stream = d->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = (unsigned)p.splits; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.splits > 1 ? 1 : 0;
  // A is K-contiguous unless it is stored transposed; B the other way round
  cudaError_t e;
  if (!trans_a && !trans_b) e = cudaLaunchKernelEx(&cfg, small_gemm_kernel<EXT, BK, GROUPS, true, false>, p);
  else if (!trans_a) e = cudaLaunchKernelEx(&cfg, small_gemm_kernel<EXT, BK, GROUPS, true, true>, p);
  else if (!trans_b) e = cudaLaunchKernelEx(&cfg, small_gemm_kernel<EXT, BK, GROUPS, false, false>, p);
  else e = cudaLaunchKernelEx(&cfg, small_gemm_kernel<EXT, BK, GROUPS, false, true>, p);
  LNN_CUDA(e);
  LNN_CHECK_LAUNCH(d);
  return LNN_OK;
}

}  // namespace

namespace lnn {

bool gemm_small_applicable(int64_t batch, int64_t m, int64_t n, int64_t k) {
  const int64_t limit = m * n * k * batch;
  return m < (1 << 24) && n < (1 << 24) && k < (1 << 24) && batch < 65536 && m * n < (1ll << 31) &&
         limit <= gemm_small_limit();
}

int gemm_small(Device* d, float* C, const float* A, const float* B, const float* bias, int64_t batch, int64_t m,
               int64_t n, int64_t k, int trans_a, int trans_b, int accumulate) {
  SmallGemm p = {};
  p.C = C; p.A = A; p.B = B; p.bias = bias;
  p.m = (int)m; p.n = (int)n; p.k = (int)k;
  p.stride_a = m * k; p.stride_b = k * n; p.stride_c = m * n;
  p.accumulate = accumulate;
  const auto aligned = [&](const float* q, int64_t ld, int64_t stride) {
    return (((uintptr_t)q) & 15) == 0 && ld % 4 == 0 && (batch == 1 || stride % 4 == 0);
  };
  p.vec_a = aligned(A, trans_a ? m : k, p.stride_a);
  p.vec_b = aligned(B, trans_b ? k : n, p.stride_b);
  p.vec_c = aligned(C, n, p.stride_c);
  const int64_t tiles64 = lnn_ceil_div(m, 64) * lnn_ceil_div(n, 64) * batch;
  const int64_t tiles32 = lnn_ceil_div(m, 32) * lnn_ceil_div(n, 32) * batch;
  // A 64 x 64 tile multiplies as much as four of 32 x 32, for rows or columns that do not exist too.  Where it is
  // half empty the small tile wins from K = 64 up, which gives its four groups a slab each (us, 64 / 32: [1, 256] x
  // [256, 1 M] 826 / 522, [1 M, 64] x [64, 4] 236 / 202, but K = 16 83 / 113); where three quarters are empty, always (4096 x
  // [16, 16] x [16, 16] 22.8 / 18.7).
  const bool wasted = 4 * tiles64 >= 4 * tiles32 || (4 * tiles64 >= 2 * tiles32 && k >= 64);
  if (tiles64 >= 2 * d->sm_count && !wasted) return launch<64, 16, 1>(d, p, (int)batch, trans_a, trans_b);
  return launch<32, 16, 4>(d, p, (int)batch, trans_a, trans_b);
}

}  // namespace lnn
