// FP64 / complex128 GEMM for the contractions of the sweep (row-major).
//
//   C[M,N] = alpha * op(A)[M,K] * op(B)[K,N] + beta * C
//
// op = N (as stored), T (transpose) or C (conjugate transpose), the three
// GemmOrder flags of the reference (cython/gemm.pxi:17-20, :21-122).  GB300
// runs FP64 on the CUDA cores only, 2 FMA per clock and SM, so a product is
// bound by how evenly its multiply-adds are spread over the SMs, not by HBM or
// by operand reuse; see k_gemm.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "kernels.cuh"
#include "tile_rules.h"

namespace cg = cooperative_groups;

namespace sm {

namespace {

// tile of the FP32 kernel k_gemm32
constexpr int BM = 64, BN = 64, BK = 16, NT = 256;

__device__ __forceinline__ double shfl_xor_T(double v, int o) {
  return __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ cplx shfl_xor_T(cplx v, int o) {
  return cplx{__shfl_xor_sync(0xffffffffu, v.re, o), __shfl_xor_sync(0xffffffffu, v.im, o)};
}

template <typename T>
__device__ __forceinline__ T load_op(const T* p, int op) {
  T v = __ldg(p);
  return op == SM_OP_C ? S<T>::conj(v) : v;
}
template <>
__device__ __forceinline__ cplx load_op<cplx>(const cplx* p, int op) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(p));
  return op == SM_OP_C ? cplx{v.x, -v.y} : cplx{v.x, v.y};
}

// One CTA (128 threads, RM x RN outputs each) per TM x TN tile and K slice; the
// slices of a tile are the CTAs of one cluster (along z), which add their partial
// tiles over DSMEM in slice order and write C once.  What bounds it: an FP64
// warp instruction holds a sub-partition's FP64 pipe for 64 clocks, so the time
// is the multiply-adds of the fullest SM.  Small tiles and up to 8 slices put
// the work of the 60..400-sized products of a split on all 152 SMs (a 64 x 64
// tile with slices of at least 64 left 18 CTAs for 174 x 174 x 190: 116 us, the
// 32 x 32 tile's 288 CTAs take 21), and the loads of a slab are in flight while the one
// before it is multiplied.  Warps whose rows all lie beyond M skip the multiply.
template <typename T, int TM, int TN, int RM, int RN>
__global__ void __launch_bounds__(128) k_gemm(int opA, int opB, int M, int N, int K, T alpha,
                                              const T* __restrict__ A, int lda,
                                              const T* __restrict__ B, int ldb, T beta,
                                              T* __restrict__ C, int ldc, int kchunk) {
  constexpr int KS = 16;                    // slab depth
  constexpr int GM = TM / RM, GN = TN / RN;  // thread grid of the tile
  static_assert(GM * GN == 128, "128 threads");
  constexpr int LA = TM * KS / 128, LB = TN * KS / 128;
  constexpr size_t kSlab = sizeof(T) * KS * (TM + 1 + TN + 1);
  constexpr size_t kTile = sizeof(T) * TM * TN;
  __shared__ __align__(16) unsigned char raw[kSlab > kTile ? kSlab : kTile];
  T(*As)[TM + 1] = reinterpret_cast<T(*)[TM + 1]>(raw);
  T(*Bs)[TN + 1] = reinterpret_cast<T(*)[TN + 1]>(raw + sizeof(T) * KS * (TM + 1));
  const int tid = threadIdx.x;
  const int tx = tid % GN, ty = tid / GN;
  // tiles along x, row by row: grid.y ends at 65535, which 16 rows a tile reach at 1 Mi
  const int tn = (N + TN - 1) / TN;
  const int m0 = (int)(blockIdx.x / tn) * TM, n0 = (int)(blockIdx.x % tn) * TN;
  T acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = S<T>::zero();
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  T ra[LA], rb[LB];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < LA; ++e) {
      const int idx = tid + e * 128;
      const int mm = opA == SM_OP_N ? idx / KS : idx % TM;
      const int kk = opA == SM_OP_N ? idx % KS : idx / TM;
      const int gm = m0 + mm, gk = k0 + kk;
      ra[e] = S<T>::zero();
      if (gm < M && gk < kend)
        ra[e] = load_op(opA == SM_OP_N ? A + (size_t)gm * lda + gk : A + (size_t)gk * lda + gm, opA);
    }
#pragma unroll
    for (int e = 0; e < LB; ++e) {
      const int idx = tid + e * 128;
      const int nn = opB == SM_OP_N ? idx % TN : idx / KS;
      const int kk = opB == SM_OP_N ? idx / TN : idx % KS;
      const int gn = n0 + nn, gk = k0 + kk;
      rb[e] = S<T>::zero();
      if (gn < N && gk < kend)
        rb[e] = load_op(opB == SM_OP_N ? B + (size_t)gk * ldb + gn : B + (size_t)gn * ldb + gk, opB);
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int e = 0; e < LA; ++e) {
      const int idx = tid + e * 128;
      As[opA == SM_OP_N ? idx % KS : idx / TM][opA == SM_OP_N ? idx / KS : idx % TM] = ra[e];
    }
#pragma unroll
    for (int e = 0; e < LB; ++e) {
      const int idx = tid + e * 128;
      Bs[opB == SM_OP_N ? idx / TN : idx % KS][opB == SM_OP_N ? idx % TN : idx / KS] = rb[e];
    }
  };
  const bool idle = m0 + (tid & ~31) / GN >= M;  // this warp's first row (the others lie below it)
  if (kbeg < kend) fetch(kbeg);
  for (int k0 = kbeg; k0 < kend; k0 += KS) {
    stage();
    __syncthreads();
    if (k0 + KS < kend) fetch(k0 + KS);
    if (!idle) {
      const int kn = min(KS, kend - k0);
#pragma unroll 4
      for (int kk = 0; kk < kn; ++kk) {
        T a[RM], b[RN];
#pragma unroll
        for (int i = 0; i < RM; ++i) a[i] = As[kk][ty + GM * i];
#pragma unroll
        for (int j = 0; j < RN; ++j) b[j] = Bs[kk][tx + GN * j];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < RN; ++j) acc[i][j] = S<T>::fma(a[i], b[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  const bool use_beta = S<T>::abs2(beta) != 0.0;
  auto put = [&](int mm, int nn, T v) {
    const int gm = m0 + mm, gn = n0 + nn;
    if (gm >= M || gn >= N) return;
    T* c = C + (size_t)gm * ldc + gn;
    T r = alpha * v;
    if (use_beta) r = S<T>::fma(beta, *c, r);
    *c = r;
  };
  const int nz = gridDim.z;
  if (nz == 1) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < RN; ++j) put(ty + GM * i, tx + GN * j, acc[i][j]);
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  T* tile = reinterpret_cast<T*>(raw);  // [TM][TN]: this slice's partial tile
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) tile[(ty + GM * i) * TN + tx + GN * j] = acc[i][j];
  cluster.sync();
  // each slice adds up its share of the tile
  const int share = (TM * TN + nz - 1) / nz;
  const int e1 = min(TM * TN, (int)(blockIdx.z + 1) * share);
  for (int e = blockIdx.z * share + tid; e < e1; e += 128) {
    T v = S<T>::zero();
    for (int z = 0; z < nz; ++z) v = v + cluster.map_shared_rank(tile, z)[e];
    put(e / TN, e % TN, v);
  }
  cluster.sync();  // no slice leaves while another reads its tile
}

// Matrix-vector shapes (N = 1, or M = 1): the Lanczos projections and norms.
// N = 1, op(A) rows contiguous (op N): block (m, kb) sums K range kb of row m
// into part[m * nkb + kb]; k_gemv_final adds the partials in order.
template <typename T>
__global__ void k_gemv_rows(int opB, const T* __restrict__ A, int lda, const T* __restrict__ B,
                            int ldb, int K, int kchunk, T* __restrict__ part) {
  __shared__ T red[32];
  const int m = blockIdx.x, kb = blockIdx.y;
  const int k0 = kb * kchunk, k1 = min(K, k0 + kchunk);
  T acc = S<T>::zero();
  for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
    const T b = load_op(opB == SM_OP_N ? B + (size_t)k * ldb : B + k, opB);
    acc = S<T>::fma(A[(size_t)m * lda + k], b, acc);
  }
  for (int o = 16; o > 0; o >>= 1) acc = acc + shfl_xor_T(acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    T t = S<T>::zero();
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t = t + red[w];
    part[(size_t)m * gridDim.y + kb] = t;
  }
}

template <typename T>
__global__ void k_gemv_final(int M, int nkb, const T* __restrict__ part, T alpha, T beta,
                             T* __restrict__ C, int ldc) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  T acc = S<T>::zero();
  for (int kb = 0; kb < nkb; ++kb) acc = acc + part[(size_t)m * nkb + kb];
  T* c = C + (size_t)m * ldc;
  *c = S<T>::abs2(beta) == 0.0 ? alpha * acc : alpha * acc + beta * *c;
}

// N = 1 with op(A) = A^T / A^H (A stored K x M) or M = 1: one thread per output
// element, the K loop coalesced across threads.
template <typename T>
__global__ void k_gemv_cols(int opA, int opB, int M, int N, int K, T alpha,
                            const T* __restrict__ A, int lda, const T* __restrict__ B, int ldb,
                            T beta, T* __restrict__ C, int ldc) {
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= (size_t)M * N) return;
  const int m = (int)(e / N), n = (int)(e % N);
  T acc = S<T>::zero();
  for (int k = 0; k < K; ++k) {
    const T a = load_op(opA == SM_OP_N ? A + (size_t)m * lda + k : A + (size_t)k * lda + m, opA);
    const T b = load_op(opB == SM_OP_N ? B + (size_t)k * ldb + n : B + (size_t)n * ldb + k, opB);
    acc = S<T>::fma(a, b, acc);
  }
  T* c = C + (size_t)m * ldc + n;
  *c = S<T>::abs2(beta) == 0.0 ? alpha * acc : alpha * acc + beta * *c;
}

template <typename T>
__global__ void k_splitk_reduce(int M, int N, int nz, const T* __restrict__ part, T alpha, T beta,
                                T* __restrict__ C, int ldc) {
  const bool use_beta = S<T>::abs2(beta) != 0.0;
  const size_t mn = (size_t)M * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < mn;
       e += (size_t)gridDim.x * blockDim.x) {
    T acc = part[e];
    for (int z = 1; z < nz; ++z) acc = acc + part[(size_t)z * mn + e];
    const int gm = (int)(e / N), gn = (int)(e % N);
    T* c = C + (size_t)gm * ldc + gn;
    T v = alpha * acc;
    if (use_beta) v = S<T>::fma(beta, *c, v);
    *c = v;
  }
}

// ---- FP32-arithmetic variant (contractions of the mixed forms) --------------
// 64 x 64 tile per CTA, 256 threads holding a 4 x 4 register tile each; operands are rounded to FP32 (complex: two FP32) when
// staged in shared memory and the products accumulate in FP32; alpha, beta
// and the output stay FP64.  Relative error ~1e-7 |A||B| per entry.
template <typename T> struct C32;
template <> struct C32<double> {
  using type = float;
  __device__ static float from(double x) { return (float)x; }
  __device__ static double to(float x) { return (double)x; }
  __device__ static float zero() { return 0.f; }
  __device__ static float fma(float a, float b, float c) { return fmaf(a, b, c); }
};
template <> struct C32<cplx> {
  using type = float2;
  __device__ static float2 from(cplx x) { return make_float2((float)x.re, (float)x.im); }
  __device__ static cplx to(float2 x) { return cplx{(double)x.x, (double)x.y}; }
  __device__ static float2 zero() { return make_float2(0.f, 0.f); }
  __device__ static float2 fma(float2 a, float2 b, float2 c) {
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
  }
};

template <typename T>
__global__ void __launch_bounds__(NT) k_gemm32(int opA, int opB, int M, int N, int K, T alpha,
                                               const T* __restrict__ A, int lda,
                                               const T* __restrict__ B, int ldb, T beta,
                                               T* __restrict__ C, int ldc, int kchunk,
                                               T* __restrict__ part) {
  using F = typename C32<T>::type;
  __shared__ F As[BK][BM + 1];
  __shared__ F Bs[BK][BN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  F acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = C32<T>::zero();
  const int kbeg = blockIdx.z * kchunk;
  const int kend = min(K, kbeg + kchunk);
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
    for (int e = 0; e < (BM * BK) / NT; ++e) {
      const int idx = tid + e * NT;
      int mm, kk;
      if (opA == SM_OP_N) { mm = idx / BK; kk = idx % BK; }
      else                { kk = idx / BM; mm = idx % BM; }
      const int gm = m0 + mm, gk = k0 + kk;
      T v = S<T>::zero();
      if (gm < M && gk < kend)
        v = opA == SM_OP_N ? load_op(A + (size_t)gm * lda + gk, opA)
                           : load_op(A + (size_t)gk * lda + gm, opA);
      As[kk][mm] = C32<T>::from(v);
    }
#pragma unroll
    for (int e = 0; e < (BN * BK) / NT; ++e) {
      const int idx = tid + e * NT;
      int nn, kk;
      if (opB == SM_OP_N) { kk = idx / BN; nn = idx % BN; }
      else                { nn = idx / BK; kk = idx % BK; }
      const int gn = n0 + nn, gk = k0 + kk;
      T v = S<T>::zero();
      if (gn < N && gk < kend)
        v = opB == SM_OP_N ? load_op(B + (size_t)gk * ldb + gn, opB)
                           : load_op(B + (size_t)gn * ldb + gk, opB);
      Bs[kk][nn] = C32<T>::from(v);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      F a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = C32<T>::fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  const bool use_beta = S<T>::abs2(beta) != 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx + 16 * j;
      if (gn >= N) continue;
      const T r = C32<T>::to(acc[i][j]);
      if (part) {
        part[(size_t)blockIdx.z * M * N + (size_t)gm * N + gn] = r;
      } else {
        T* c = C + (size_t)gm * ldc + gn;
        T v = alpha * r;
        if (use_beta) v = S<T>::fma(beta, *c, v);
        *c = v;
      }
    }
  }
}

}  // namespace

namespace {

template <typename T, int TM, int TN, int RM, int RN>
int launch_gemm(cudaStream_t st, int opA, int opB, int M, int N, int K, T alpha, const T* A, int lda,
                const T* B, int ldb, T beta, T* C, int ldc, int nz) {
  const int kchunk = ((K + nz - 1) / nz + 15) / 16 * 16;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((size_t)((N + TN - 1) / TN) * ((M + TM - 1) / TM)), 1, nz);
  cfg.blockDim = dim3(128);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = nz;
  cfg.attrs = attr;
  cfg.numAttrs = nz > 1 ? 1 : 0;
  SM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_gemm<T, TM, TN, RM, RN>, opA, opB, M, N, K, alpha, A, lda,
                                   B, ldb, beta, C, ldc, kchunk));
  note_launch();
  return SM_OK;
}

}  // namespace

namespace {
template <typename T>
int gemm(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, T alpha, const T* A,
         int lda, const T* B, int ldb, T beta, T* C, int ldc) {
  const int sms = std::max(1, ctx.num_sms);
  if (M < 0 || N < 0 || K < 0) {
    set_error("gemm: negative size");
    return SM_ERR_VALUE;
  }
  if (M == 0 || N == 0) return SM_OK;
  if (K == 0) {
    // C = beta C  (or zero)
    return scale_matrix<T>(st, M, N, beta, C, ldc);
  }
  if (M > 65535 * BM) {  // the rows of the FP32 kernel's grid: one limit for all forms
    set_error("gemm: M too large");
    return SM_ERR_VALUE;
  }
  const GemmCut cut = gemm_cut(M, N, K, sizeof(T) != sizeof(double), sms);
  if (cut.tile == 16)
    return launch_gemm<T, 16, 16, 1, 2>(st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc,
                                        cut.slices);
  return launch_gemm<T, 32, 32, 2, 4>(st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc,
                                      cut.slices);
}
}  // namespace

// K slices of the FP32 kernel for an M x N x K product on `sms` SMs: enough CTAs
// for about two waves, each slice at least 64 deep; 1 = no split.
int splitk_slices(int M, int N, int K, int sms) {
  const long tiles = (long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  if (tiles >= sms || K < 128) return 1;
  const long want = (2L * sms + tiles - 1) / tiles;
  return (int)std::max(1L, std::min({want, (long)(K / 64), 32L}));
}

template <typename T>
int gemm_ctx(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, T alpha, const T* A,
             int lda, const T* B, int ldb, T beta, T* C, int ldc) {
  return gemm_ctx_sel(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, true);
}

namespace {
// Whether a product in BF16 slices (two launches, three for a complex one) is faster
// than the FP64 kernel.  A mixed split of 128 rows, products of 128^3, takes 0.87 ms
// with slices and 0.78 without; an Euler step takes 90.0 ms with slices from 150^3 on
// and 92.6 from 180^3 on.  Complex: 96 rows 0.94 ms with and 0.85 without, 128 rows
// 1.09 and 1.16.
template <typename T>
bool slices_pay(int M, int N, int K) {
  const double mnk = (double)M * N * K;
  if constexpr (sizeof(T) == sizeof(double)) return mnk >= 3.5e6 && gemm_oz_eligible(M, N, K);
  return mnk >= 1.6e6 && gemm_cplx_oz_eligible(M, N, K);
}
}  // namespace

template <typename T>
int gemm_ctx_sel(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, T alpha,
                 const T* A, int lda, const T* B, int ldb, T beta, T* C, int ldc, bool allow_tc) {
  if (M == 0 || N == 0 || K == 0) return gemm<T>(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  if constexpr (sizeof(T) == sizeof(double)) {
    // mixed forms: FP64-accurate products on the BF16 tensor cores
    if (allow_tc && ctx.precision != SM_PRECISION_FP64 && ctx.fp64_tc && slices_pay<T>(M, N, K)) {
      ctx.stats.gemm_oz_launches += 1;
      ctx.stats.gemm_oz_flops += 2.0 * M * N * K;
      if (ctx.timing) SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
      SM_CHECK(gemm_oz(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc));
      if (ctx.timing) {
        SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
        SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
        float ms = 0.f;
        SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
        ctx.stats.gemm_oz_ms += ms;
      }
      return SM_OK;
    }
  } else {
    // mixed forms, complex operands: three real FP64-accurate products (3M)
    if (allow_tc && ctx.precision != SM_PRECISION_FP64 && ctx.fp64_tc && slices_pay<T>(M, N, K)) {
      ctx.stats.gemm_oz_launches += 3;
      ctx.stats.gemm_oz_flops += 6.0 * M * N * K;
      if (ctx.timing) SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
      SM_CHECK(gemm_cplx_3m(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc,
                            true));
      if (ctx.timing) {
        SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
        SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
        float ms = 0.f;
        SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
        ctx.stats.gemm_oz_ms += ms;
      }
      return SM_OK;
    }
  }
  ctx.stats.gemm_launches += 1;
  ctx.stats.gemm_flops += 2.0 * M * N * K * (sizeof(T) == sizeof(double) ? 1.0 : 4.0);
  if (N == 1 && opA == SM_OP_N && K >= 1024 && M <= 65535) {
    // long dot products: K split over blocks, partials summed in order
    const int nkb = std::min(64, (K + 4095) / 4096);
    const int kchunk = (K + nkb - 1) / nkb;
    T* part;
    SM_CHECK(ctx.scratch("gemv.part", (size_t)M * nkb, &part));
    k_gemv_rows<T><<<dim3(M, nkb), 256, 0, st>>>(opB, A, lda, B, ldb, K, kchunk, part);
    k_gemv_final<T><<<(M + 127) / 128, 128, 0, st>>>(M, nkb, part, alpha, beta, C, ldc);
    note_launch(2);
    SM_CUDA_CHECK(cudaGetLastError());
    return SM_OK;
  }
  if ((N == 1 || M == 1) && K <= 4096) {
    const size_t mn = (size_t)M * N;
    k_gemv_cols<T><<<(unsigned)((mn + 127) / 128), 128, 0, st>>>(opA, opB, M, N, K, alpha, A, lda,
                                                                   B, ldb, beta, C, ldc);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
    return SM_OK;
  }
  auto run = [&]() -> int {
    return gemm<T>(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  };
  if (!ctx.timing) return run();
  SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
  SM_CHECK(run());
  SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
  SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
  float ms = 0.f;
  SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
  ctx.stats.gemm_ms += ms;
  return SM_OK;
}

template <typename T>
int gemm_ctx_f32(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, T alpha,
                 const T* A, int lda, const T* B, int ldb, T beta, T* C, int ldc) {
  if (M == 0 || N == 0 || K == 0) return gemm<T>(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  ctx.stats.gemm32_launches += 1;
  ctx.stats.gemm32_flops += 2.0 * M * N * K * (sizeof(T) == sizeof(double) ? 1.0 : 4.0);
  if constexpr (sizeof(T) == sizeof(double)) {
    if (gemm_tc_eligible(M, N, K)) {
      if (ctx.timing) SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
      SM_CHECK(gemm_tc(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc));
      ctx.stats.gemm_tc_launches += 1;
      ctx.stats.gemm_tc_flops += 2.0 * M * N * K;
      if (ctx.timing) {
        SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
        SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
        float ms = 0.f;
        SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
        ctx.stats.gemm32_ms += ms;
        ctx.stats.gemm_tc_ms += ms;
      }
      return SM_OK;
    }
  } else {
    // complex operands: three real 3xTF32 products on split planes (3M)
    if (gemm_cplx_tc_eligible(M, N, K)) {
      if (ctx.timing) SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
      SM_CHECK(gemm_cplx_3m(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc,
                            false));
      ctx.stats.gemm_tc_launches += 3;
      ctx.stats.gemm_tc_flops += 6.0 * M * N * K;
      if (ctx.timing) {
        SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
        SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
        float ms = 0.f;
        SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
        ctx.stats.gemm32_ms += ms;
        ctx.stats.gemm_tc_ms += ms;
      }
      return SM_OK;
    }
  }
  // FP32 runs 64x the FP64 rate: split K only when the output has very few tiles
  const int nz = splitk_slices(M, N, K, std::max(1, ctx.num_sms) / 2);
  T* part = nullptr;
  if (nz > 1) SM_CHECK(ctx.scratch("gemm.splitk", (size_t)nz * M * N, &part));
  const int kchunk = nz > 1 ? ((K + nz - 1) / nz + BK - 1) / BK * BK : K;
  const int nzz = nz > 1 ? (K + kchunk - 1) / kchunk : 1;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, nzz);
  if (grid.y > 65535) {
    set_error("gemm: M too large");
    return SM_ERR_VALUE;
  }
  if (ctx.timing) SM_CUDA_CHECK(cudaEventRecord(ctx.ev0, st));
  k_gemm32<T><<<grid, NT, 0, st>>>(opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk,
                                   nzz > 1 ? part : nullptr);
  note_launch();
  SM_CUDA_CHECK(cudaGetLastError());
  if (nzz > 1) {
    const size_t mn = (size_t)M * N;
    const int blocks = (int)std::min<size_t>((mn + 255) / 256, 4096);
    k_splitk_reduce<T><<<blocks, 256, 0, st>>>(M, N, nzz, part, alpha, beta, C, ldc);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
  }
  if (ctx.timing) {
    SM_CUDA_CHECK(cudaEventRecord(ctx.ev1, st));
    SM_CUDA_CHECK(cudaEventSynchronize(ctx.ev1));
    float ms = 0.f;
    SM_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1));
    ctx.stats.gemm32_ms += ms;
  }
  return SM_OK;
}

template int gemm_ctx_f32<double>(Ctx&, cudaStream_t, int, int, int, int, int, double,
                                  const double*, int, const double*, int, double, double*, int);
template int gemm_ctx_f32<cplx>(Ctx&, cudaStream_t, int, int, int, int, int, cplx, const cplx*,
                                int, const cplx*, int, cplx, cplx*, int);

template int gemm_ctx<double>(Ctx&, cudaStream_t, int, int, int, int, int, double, const double*,
                              int, const double*, int, double, double*, int);
template int gemm_ctx_sel<double>(Ctx&, cudaStream_t, int, int, int, int, int, double,
                                  const double*, int, const double*, int, double, double*, int,
                                  bool);
template int gemm_ctx_sel<cplx>(Ctx&, cudaStream_t, int, int, int, int, int, cplx, const cplx*,
                                int, const cplx*, int, cplx, cplx*, int, bool);
template int gemm_ctx<cplx>(Ctx&, cudaStream_t, int, int, int, int, int, cplx, const cplx*, int,
                            const cplx*, int, cplx, cplx*, int);

}  // namespace sm
