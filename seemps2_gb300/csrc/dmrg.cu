// Two-site effective-Hamiltonian matvec of DMRG (the reference's
// QuadraticForm.two_site_operator._matvec, operators/quadratic.py:187-237):
//
//   out[a, ko, lo, g] = sum_{b,c,d,k,l,f} L[a, c, b] v[b, k, l, f] H[c, ko, k, lo, l, d] R[g, d, f]
//
// with L (bra bond a, MPO bond c, ket bond b), the two-site MPO H = O_i O_{i+1}
// (_contract_last_and_first) and R (bra g, MPO d, ket f).  Three steps:
//   1. X1[(a,c), (k,l,f)] = L[(a,c), b] v[b, (k,l,f)]            GEMM, 2 a c b k l f flops
//   2. X2[a, ko, lo, d, f] = sum_{c,k,l} X1[a,c,k,l,f] H[c,ko,k,lo,l,d]
//                                                               k_h12_apply, 2 a f (c k l)(ko lo d)
//   3. out[(a,ko,lo), g] = X2[(a,ko,lo), (d,f)] R[g, (d,f)]^T   GEMM reading R in place (op T)
// At chi = 256, D = 5, d = 2: 671 + 52 + 671 MFLOP.  The precision argument
// picks the products: FP64 SIMT, FP64-accurate on the BF16 tensor cores,
// FP32-accurate 3xTF32, or one BF16 product with FP32 accumulation (the
// precision pattern of the DMRG configuration); complex operands use the SIMT
// kernels (FP64, or FP32 for the two reduced precisions).
#include <algorithm>

#include "kernels.cuh"

namespace sm {

namespace {

// One pass of the two-site MPO over a block's outputs: block (32, 8) takes 32 values
// of f, 8 of a, one (ko, lo) and up to kH12Out values of dd; thread (f, a) gets the
// sums acc[dd] = sum_{c,k,l} H[c][ko][k][lo][l][dd] X1[a][c][k][l][f] in that order.
// The nonzero entries of each output are listed in shared memory first (warp w lists
// output w, chunks of kH12In inputs): a bulk site of the Heisenberg chain has 36 of 400,
// and testing each entry where it is used cost more than everything else (an FP64
// comparison holds the FP64 pipe for 64 clocks; at a = f = 108, D = 5 96 us, in FP32 at
// 256 56 us).  Bound by the traffic of X1 and X2 through L2.
constexpr int kH12Out = 8, kH12In = 256;
template <typename T, typename V>
struct H12Shared {
  V h[kH12Out][kH12In];
  short in[kH12Out][kH12In];
  int cnt[kH12Out];
};
__device__ __forceinline__ bool h12_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool h12_zero(double x) { return x == 0.0; }
__device__ __forceinline__ bool h12_zero(cplx x) { return x.re == 0.0 && x.im == 0.0; }
template <typename T>
__device__ __forceinline__ void h12_put(T& d, T x) { d = x; }
__device__ __forceinline__ void h12_put(float& d, double x) { d = (float)x; }
template <typename T>
__device__ __forceinline__ T h12_fma(T h, T x, T acc) { return S<T>::fma(h, x, acc); }
__device__ __forceinline__ float h12_fma(float h, float x, float acc) { return fmaf(h, x, acc); }

template <typename T, typename V>
__device__ __forceinline__ void h12_sums(const V* __restrict__ X1, const T* __restrict__ H, int A,
                                         int Cc, int p1, int p2, int E, int F, int ko, int lo,
                                         int d0, int nd, int a, int f, V (&acc)[kH12Out],
                                         H12Shared<T, V>& sh) {
  const int nin = Cc * p1 * p2;
  const int warp = threadIdx.y, lane = threadIdx.x;
  const bool on = a < A && f < F;
  const V* x = X1 + (size_t)(on ? a : 0) * nin * F + (on ? f : 0);
  for (int i0 = 0; i0 < nin; i0 += kH12In) {
    const int ni = min(kH12In, nin - i0);
    __syncthreads();  // the previous chunk has been used
    if (warp < nd) {
      int n = 0;
      for (int j = 0; j < ni; j += 32) {
        const int i = i0 + j + lane;
        bool put = false;
        V h{};
        if (j + lane < ni) {
          const int c = i / (p1 * p2), k = i / p2 % p1, l = i % p2;
          h12_put(h, H[((((size_t)(c * p1 + ko) * p1 + k) * p2 + lo) * p2 + l) * E + d0 + warp]);
          put = !h12_zero(h);  // as multiplied: 1e-60 is zero in FP32
        }
        const unsigned m = __ballot_sync(0xffffffffu, put);
        if (put) {
          const int at = n + __popc(m & ((1u << lane) - 1u));
          sh.h[warp][at] = h;
          sh.in[warp][at] = (short)(j + lane);
        }
        n += __popc(m);
      }
      if (lane == 0) sh.cnt[warp] = n;
    }
    __syncthreads();
    const V* xc = x + (size_t)i0 * F;
#pragma unroll
    for (int d = 0; d < kH12Out; ++d) {
      if (d >= nd) break;
      const int n = sh.cnt[d];
      for (int i = 0; i < n; ++i)
        if (on) acc[d] = h12_fma(sh.h[d][i], xc[(size_t)sh.in[d][i] * F], acc[d]);
    }
  }
}
inline dim3 h12_grid(int a, int p1, int p2, int e, int f) {
  return dim3((f + 31) / 32, (a + 7) / 8, p1 * p2 * ((e + kH12Out - 1) / kH12Out));
}

// X2[a][ko][lo][dd][f] = sum_{c,k,l} X1[a][c][k][l][f] H[c][ko][k][lo][l][dd].
template <typename T>
__global__ void __launch_bounds__(256) k_h12_apply(const T* __restrict__ X1, const T* __restrict__ H,
                                                   int A, int Cc, int p1, int p2, int E, int F,
                                                   T* __restrict__ X2) {
  __shared__ H12Shared<T, T> sh;
  const int nch = (E + kH12Out - 1) / kH12Out, kl = blockIdx.z / nch;
  const int d0 = blockIdx.z % nch * kH12Out, nd = min(kH12Out, E - d0);
  const int f = blockIdx.x * 32 + threadIdx.x, a = blockIdx.y * 8 + threadIdx.y;
  T acc[kH12Out];
#pragma unroll
  for (int d = 0; d < kH12Out; ++d) acc[d] = S<T>::zero();
  h12_sums<T, T>(X1, H, A, Cc, p1, p2, E, F, kl / p2, kl % p2, d0, nd, a, f, acc, sh);
  if (a >= A || f >= F) return;
  T* out = X2 + (((size_t)a * p1 * p2 + kl) * E + d0) * F + f;
#pragma unroll
  for (int d = 0; d < kH12Out; ++d)
    if (d < nd) out[(size_t)d * F] = acc[d];
}

template <typename T>
int product(Ctx& ctx, cudaStream_t st, int precision, int opA, int opB, int M, int N, int K,
            const T* A, int lda, const T* B, int ldb, T* C, int ldc) {
  const T one = S<T>::one(), zero = S<T>::zero();
  if constexpr (sizeof(T) == sizeof(double)) {
    if (precision == SM_MATVEC_FP64TC && gemm_oz_eligible(M, N, K)) {
      ctx.stats.gemm_oz_launches += 1;
      ctx.stats.gemm_oz_flops += 2.0 * M * N * K;
      return gemm_oz(ctx, st, opA, opB, M, N, K, one, A, lda, B, ldb, zero, C, ldc);
    }
    if ((precision == SM_MATVEC_TF32X3 || precision == SM_MATVEC_BF16) &&
        gemm_tc_eligible(M, N, K)) {
      ctx.stats.gemm_tc_launches += 1;
      ctx.stats.gemm_tc_flops += 2.0 * M * N * K;
      return gemm_tc(ctx, st, opA, opB, M, N, K, one, A, lda, B, ldb, zero, C, ldc,
                     precision == SM_MATVEC_BF16);
    }
  }
  if (precision == SM_MATVEC_TF32X3 || precision == SM_MATVEC_BF16)
    return gemm_ctx_f32<T>(ctx, st, opA, opB, M, N, K, one, A, lda, B, ldb, zero, C, ldc);
  return gemm_ctx_sel<T>(ctx, st, opA, opB, M, N, K, one, A, lda, B, ldb, zero, C, ldc, false);
}

}  // namespace

template <typename T>
int two_site_matvec(Ctx& ctx, cudaStream_t st, int a, int c, int b, int p1, int p2, int e, int g,
                    int f, const T* L, const T* H, const T* R, const T* v, T* out, int precision) {
  T *X1, *X2;
  SM_CHECK(ctx.scratch("mv.X1", (size_t)a * c * p1 * p2 * f, &X1));
  SM_CHECK(ctx.scratch("mv.X2", (size_t)a * p1 * p2 * e * f, &X2));
  SM_CHECK(product<T>(ctx, st, precision, SM_OP_N, SM_OP_N, a * c, p1 * p2 * f, b, L, b, v,
                      p1 * p2 * f, X1, p1 * p2 * f));
  // FP64 arithmetic at every precision: the intermediates are FP64, and
  // converting them to FP32 costs GB300's FP64 pipe as much as the FMAs
  k_h12_apply<T><<<h12_grid(a, p1, p2, e, f), dim3(32, 8), 0, st>>>(X1, H, a, c, p1, p2, e, f, X2);
  note_launch();
  SM_CUDA_CHECK(cudaGetLastError());
  return product<T>(ctx, st, precision, SM_OP_N, SM_OP_T, a * p1 * p2, g, e * f, X2, e * f, R,
                    e * f, out, g);
}

template int two_site_matvec<double>(Ctx&, cudaStream_t, int, int, int, int, int, int, int, int,
                                     const double*, const double*, const double*, const double*,
                                     double*, int);
template int two_site_matvec<cplx>(Ctx&, cudaStream_t, int, int, int, int, int, int, int, int,
                                   const cplx*, const cplx*, const cplx*, const cplx*, cplx*, int);

// ---------------------------------------------------------------------------
// Prepared form for a Lanczos run (real operands, TF32X3 / BF16): L and R do
// not change between matvecs, so they become tensor-core operand planes once.
// Per matvec only v is converted; the first product writes X1 in FP32, the
// MPO step reads it in FP32 and writes X2 straight into the second product's
// operand planes, and the second product writes the FP64 result.
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ float tf32_round(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// X2[(a, ko, lo)][(dd, f)] = sum_{c,k,l} X1[a][c][k][l][f] H[c][ko][k][lo][l][dd]
// in FP32, written as K-contiguous operand rows of kp entries (the caller
// zeroes the columns past E F): one BF16 plane, or TF32 hi = rna(x) and
// lo = x - hi.  Blocks as k_h12_apply's; H (FP64) is converted as it is listed.
template <bool BF16>
__global__ void __launch_bounds__(256)
    k_h12_planes(const float* __restrict__ X1, const double* __restrict__ H, int A, int Cc, int p1,
                 int p2, int E, int F, int kp, void* __restrict__ hi, float* __restrict__ lo) {
  __shared__ H12Shared<double, float> sh;
  const int nch = (E + kH12Out - 1) / kH12Out, kl = blockIdx.z / nch;
  const int d0 = blockIdx.z % nch * kH12Out, nd = min(kH12Out, E - d0);
  const int f = blockIdx.x * 32 + threadIdx.x, a = blockIdx.y * 8 + threadIdx.y;
  float acc[kH12Out];
#pragma unroll
  for (int d = 0; d < kH12Out; ++d) acc[d] = 0.f;
  h12_sums<double, float>(X1, H, A, Cc, p1, p2, E, F, kl / p2, kl % p2, d0, nd, a, f, acc, sh);
  if (a >= A || f >= F) return;
  const size_t row = ((size_t)a * p1 * p2 + kl) * kp + (size_t)d0 * F + f;
#pragma unroll
  for (int d = 0; d < kH12Out; ++d) {
    if (d >= nd) break;
    const size_t o = row + (size_t)d * F;
    if (BF16) {
      reinterpret_cast<__nv_bfloat16*>(hi)[o] = __float2bfloat16_rn(acc[d]);
    } else {
      const float h = tf32_round(acc[d]);
      reinterpret_cast<float*>(hi)[o] = h;
      lo[o] = acc[d] - h;
    }
  }
}

}  // namespace

int two_site_prepare(Ctx& ctx, cudaStream_t st, int a, int c, int b, int p1, int p2, int e,
                     int g, int f, const double* L, const double* R, int precision) {
  if (precision != SM_MATVEC_TF32X3 && precision != SM_MATVEC_BF16) {
    set_error("two_site_prepare: the prepared matvec takes SM_MATVEC_TF32X3 or SM_MATVEC_BF16");
    return SM_ERR_VALUE;
  }
  MatvecPrep& mp = ctx.mvp;
  mp = MatvecPrep{};
  mp.precision = precision;
  mp.a = a, mp.c = c, mp.b = b, mp.p1 = p1, mp.p2 = p2, mp.e = e, mp.g = g, mp.f = f;
  mp.L = L;
  mp.R = R;
  const int n1 = p1 * p2 * f;
  mp.tc = gemm_tc_eligible(a * c, n1, b) && gemm_tc_eligible(a * p1 * p2, g, e * f);
  if (!mp.tc) return SM_OK;  // small shapes: the matvec runs the generic path
  const bool bf16 = precision == SM_MATVEC_BF16;
  const int TK = tc_kslab(bf16);
  mp.kpL = (b + TK - 1) / TK * TK;
  mp.kpR = (e * f + TK - 1) / TK * TK;
  const size_t es = bf16 ? 2 : 4;
  SM_CHECK(ctx.scratch("mvp.Lh", es * (size_t)a * c * mp.kpL, &mp.Lh));
  SM_CHECK(ctx.scratch("mvp.Rh", es * (size_t)g * mp.kpR, &mp.Rh));
  if (!bf16) {
    SM_CHECK(ctx.scratch("mvp.Ll", (size_t)a * c * mp.kpL, &mp.Ll));
    SM_CHECK(ctx.scratch("mvp.Rl", (size_t)g * mp.kpR, &mp.Rl));
  }
  // L[(a,c)][b] and R[g][(d,f)] are K-contiguous already
  SM_CHECK(tc_planes(ctx, st, L, b, a * c, b, mp.kpL, 0, bf16, mp.Lh, mp.Ll));
  SM_CHECK(tc_planes(ctx, st, R, e * f, g, e * f, mp.kpR, 0, bf16, mp.Rh, mp.Rl));
  return SM_OK;
}

int two_site_matvec_prepared(Ctx& ctx, cudaStream_t st, const double* H, const double* v,
                             double* out) {
  const MatvecPrep& mp = ctx.mvp;
  if (mp.precision < 0) {
    set_error("two_site_matvec_prepared: no prepared operator (sm_two_site_prepare)");
    return SM_ERR_VALUE;
  }
  const int a = mp.a, c = mp.c, b = mp.b, p1 = mp.p1, p2 = mp.p2, e = mp.e, g = mp.g, f = mp.f;
  if (!mp.tc)
    return two_site_matvec<double>(ctx, st, a, c, b, p1, p2, e, g, f, mp.L, H, mp.R, v, out,
                                   mp.precision);
  const bool bf16 = mp.precision == SM_MATVEC_BF16;
  const size_t es = bf16 ? 2 : 4;
  const int n1 = p1 * p2 * f, m3 = a * p1 * p2;
  void *vh, *x2h;
  float *vl = nullptr, *x2l = nullptr, *X1;
  SM_CHECK(ctx.scratch("mvp.vh", es * (size_t)n1 * mp.kpL, &vh));
  SM_CHECK(ctx.scratch("mvp.x2h", es * (size_t)m3 * mp.kpR, &x2h));
  SM_CHECK(ctx.scratch("mvp.X1", (size_t)a * c * n1, &X1));
  if (!bf16) {
    SM_CHECK(ctx.scratch("mvp.vl", (size_t)n1 * mp.kpL, &vl));
    SM_CHECK(ctx.scratch("mvp.x2l", (size_t)m3 * mp.kpR, &x2l));
  }
  // v[b][(k,l,f)]: op(B)^T rows are its columns
  SM_CHECK(tc_planes(ctx, st, v, n1, n1, b, mp.kpL, 1, bf16, vh, vl));
  ctx.stats.gemm_tc_launches += 2;
  ctx.stats.gemm_tc_flops += 2.0 * a * c * n1 * b + 2.0 * m3 * g * e * f;
  SM_CHECK(gemm_tc_planes<float>(ctx, st, a * c, n1, mp.kpL, bf16, mp.Lh, mp.Ll, vh, vl, 1.0,
                                 0.0, X1, n1));
  if (mp.kpR > e * f) {  // zero K padding of the second product's A operand
    SM_CUDA_CHECK(cudaMemsetAsync(x2h, 0, es * (size_t)m3 * mp.kpR, st));
    if (!bf16) SM_CUDA_CHECK(cudaMemsetAsync(x2l, 0, sizeof(float) * (size_t)m3 * mp.kpR, st));
  }
  const dim3 grd = h12_grid(a, p1, p2, e, f);
  if (bf16)
    k_h12_planes<true><<<grd, dim3(32, 8), 0, st>>>(X1, H, a, c, p1, p2, e, f, mp.kpR, x2h, x2l);
  else
    k_h12_planes<false><<<grd, dim3(32, 8), 0, st>>>(X1, H, a, c, p1, p2, e, f, mp.kpR, x2h, x2l);
  note_launch();
  SM_CUDA_CHECK(cudaGetLastError());
  return gemm_tc_planes<double>(ctx, st, m3, g, mp.kpR, bf16, x2h, x2l, mp.Rh, mp.Rl, 1.0, 0.0,
                                out, g);
}

}  // namespace sm
