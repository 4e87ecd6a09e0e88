// FP64 orthogonalisation of rows through an FP32 start (the plain FP64 splits).
//
// svd_split needs X R with X unitary and the rows of X R orthogonal to FP64
// level (the one-sided Jacobi's result).  The FP64 Jacobi of svd.cu reaches it
// in 8..12 sweeps of k - 1 rounds, and each round costs a grid barrier and a
// trip through L2 (~4 us) whatever its arithmetic: 12 ms on a 174 x 190 matrix
// whose FP64 work is 0.1 ms of the chip's FP64 rate.  Here, following the
// mixed-precision Jacobi SVD of Gao, Ma and Shao (arXiv 2209.04626), an FP32
// SVD supplies X to FP32 accuracy and FP64 matrix products do the rest:
//
//   1. the FP32 stage (svd_cluster_*.cu) factors R^T; its rows are
//      s_i u_i^T, so their normalised conjugates are X0 ~ U^H;
//   2. Newton-Schulz steps X <- (1.5 I - 0.5 X X^H) X make X unitary to FP64
//      rounding (X0 is off by ~1e-6: two steps), and W = X R is then an exact
//      unitary transform of R whatever the quality of X0;
//   3. correction steps: from G = W W^H the anti-Hermitian E of first-order
//      rotation angles, E_ij = G_ij / (G_ii - G_jj) for every pair that the
//      Jacobi's own test would still rotate, and W <- exp(E) W by its Taylor
//      series, cut where the next term is below rounding (|E|_inf is read back
//      with the test's verdict).  Each step squares the overlaps of separated
//      pairs: usually two steps and one closing test;
//   4. where pairs are left whose angle is not small (singular values below
//      the FP32 resolution of the first pass, nearly equal ones), the FP32
//      stage runs again on the graded W (up to three times), where it takes one
//      or two sweeps and resolves the next 5..6 decades; what is left after that
//      is the FP64 Jacobi's, which starts from W and needs few sweeps.
//
// The closing test is the Jacobi's convergence test on every pair of rows, so
// a caller that gets `converged` needs no Jacobi at all.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "kernels.cuh"

namespace sm {

namespace {

constexpr double kAngleMax = 1e-2;   // largest angle a correction step takes
constexpr double kAngleSafe = 1e-3;  // ... before another FP32 pass (larger ones are noise then)
constexpr double kAngleInf = 0.05;   // |E|_inf above which the FP32 stage runs again
constexpr double kDevDone = 2e-8;    // |X X^H - I|_inf that one Newton-Schulz step takes to rounding
constexpr double kDevMax = 0.9;      // largest entry of X X^H - I from which no step is tried
// Newton-Schulz steps at most after the first: nearly parallel rows (an entry of 0.9) are
// eleven steps from rounding.  Of 488 splits in eight chains of bond 256, 42 went to the
// FP64 Jacobi with eight steps (~19 ms each against 0.1 a step), 38 with twelve.
constexpr int kNewtonSteps = 12;
constexpr int kLevels = 4;           // FP32 passes at most
constexpr int kSteps = 12;           // correction steps at most
constexpr int kTaylor = 8;           // terms of exp(E) at most

// What the host reads after a test.
struct PrecondStat {
  double dev;           // |X X^H - I|_inf before the last Newton-Schulz step
  double entry;         // and its largest entry
  double einf;          // largest row sum of |E|
  unsigned int viol;    // pairs that the Jacobi would rotate
  unsigned int left;    // ... of them without a small angle
  int status;           // of the FP32 stage
  int missing;          // rows of zero norm among X0's
};

// X0 from the FP32 stage: block b takes its row b of `cap`, finds the row's place
// in descending order of norm (ties by index) and writes the normalised
// conjugate there if the place is below k.
template <typename T>
__global__ void __launch_bounds__(128) k_rows_to_basis(const T* __restrict__ rows,
                                                       const double* __restrict__ nrm, int cap,
                                                       int k, const JacobiCtl* ctl,
                                                       T* __restrict__ X, PrecondStat* stat) {
  __shared__ int place;
  const int b = blockIdx.x;
  if (threadIdx.x == 0) place = 0;
  __syncthreads();
  const double nb = nrm[b];
  int n = 0;
  for (int j = threadIdx.x; j < cap; j += blockDim.x) {
    const double nj = nrm[j];
    n += (nj > nb) || (nj == nb && j < b);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(&place, n);
  __syncthreads();
  const int p = place;
  if (b == 0 && threadIdx.x == 0) stat->status = ctl->status;
  if (p >= k) return;
  const double inv = nb > 0.0 ? 1.0 / nb : 0.0;
  if (threadIdx.x == 0 && !(nb > 0.0)) atomicAdd(&stat->missing, 1);
  for (int x = threadIdx.x; x < k; x += blockDim.x)
    X[(size_t)p * k + x] = S<T>::scale(S<T>::conj(rows[(size_t)b * k + x]), inv);
}

// M <- 1.5 I - 0.5 M, the Newton-Schulz factor of M = X X^H: block i takes row i; the
// largest row sum and entry of |M - I| go to *stat.  The row sum says when to stop: it
// bounds the spectral deviation, which the largest entry does not (k entries of 2e-8 in
// phase are one of k 2e-8, whose square a step leaves behind).
template <typename T>
__global__ void __launch_bounds__(128) k_newton_schulz(T* M, int k, PrecondStat* stat) {
  __shared__ double red[4], top[4];
  const int i = blockIdx.x;
  double sum = 0.0, worst = 0.0;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    T& m = M[(size_t)i * k + j];
    const T d = i == j ? m - S<T>::one() : m;
    const double a = sqrt(S<T>::abs2(d));
    sum += a;
    worst = a > worst ? a : worst;  // a NaN shows in the sum
    m = S<T>::scale(d, -0.5);
    if (i == j) m = m + S<T>::one();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const double a = __shfl_xor_sync(0xffffffffu, worst, o);
    worst = a > worst ? a : worst;
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = sum;
    top[threadIdx.x >> 5] = worst;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 4; ++w) worst = top[w] > worst ? top[w] : worst;
  // without its sign bit a NaN counts as the largest
  auto most = [](double* at, double x) {
    atomicMax(reinterpret_cast<unsigned long long*>(at),
              (unsigned long long)__double_as_longlong(fabs(x)));
  };
  most(&stat->dev, red[0] + red[1] + red[2] + red[3]);
  most(&stat->entry, worst);
}

// E and the verdict from G = W W^H: block i takes row i.  The test is the
// Jacobi's (k_jacobi): rows of squared norm at most defl_rel |W|^2 take no part,
// a pair is orthogonal if |g|^2 <= tol2 a b, or below the rounding floor.
template <typename T>
__global__ void __launch_bounds__(128) k_angles(const T* __restrict__ G, int k, int l, double tol2,
                                                int use_floor, double defl_rel, double amax,
                                                T* __restrict__ E, PrecondStat* stat) {
  __shared__ double red[4];
  __shared__ int cnt[2];
  const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  double f = 0.0;
  for (int j = threadIdx.x; j < k; j += blockDim.x) f += S<T>::real(G[(size_t)j * k + j]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
  if (lane == 0) red[warp] = f;
  __syncthreads();
  const double frob2 = red[0] + red[1] + red[2] + red[3];
  __syncthreads();
  const double thr = defl_rel * frob2;
  double tiny2 = 0.0;
  if (use_floor) {
    const double tiny = 16.0 * l * DBL_EPSILON * DBL_EPSILON * frob2;
    tiny2 = tiny * tiny;
  }
  const double a = S<T>::real(G[(size_t)i * k + i]);
  double sum = 0.0;
  int viol = 0, left = 0;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    // the pair's lower entry decides for both, so that E is anti-Hermitian exactly
    const T g = i >= j ? G[(size_t)i * k + j] : S<T>::conj(G[(size_t)j * k + i]);
    const double b = S<T>::real(G[(size_t)j * k + j]);
    const double g2 = S<T>::abs2(g);
    T e = S<T>::zero();
    if (i != j && a > thr && b > thr && !(g2 <= tiny2) && !(g2 <= tol2 * a * b)) {
      const double d = a - b;
      ++viol;
      if (g2 <= amax * amax * d * d) {
        e = S<T>::scale(g, 1.0 / d);
        sum += sqrt(g2) / fabs(d);
      } else {
        ++left;
      }
    }
    E[(size_t)i * k + j] = e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    viol += __shfl_xor_sync(0xffffffffu, viol, o);
    left += __shfl_xor_sync(0xffffffffu, left, o);
  }
  if (lane == 0) {
    red[warp] = sum;
    if (viol) atomicAdd(&cnt[0], viol);
    if (left) atomicAdd(&cnt[1], left);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double s = red[0] + red[1] + red[2] + red[3];
    if (s > 0.0)
      atomicMax(reinterpret_cast<unsigned long long*>(&stat->einf),
                (unsigned long long)__double_as_longlong(s));
    if (cnt[0]) atomicAdd(&stat->viol, (unsigned int)cnt[0]);
    if (cnt[1]) atomicAdd(&stat->left, (unsigned int)cnt[1]);
  }
}

}  // namespace

template <typename T>
bool precondition_takes(Ctx& ctx, int k, int l) {
  return k >= kPrecondMinRows && split_cluster_fits<T>(ctx, l, k);
}

template <typename T>
int precondition_rows(Ctx& ctx, cudaStream_t st, T* R, int k, int l, double tol2, int use_floor,
                      double defl_rel, bool* converged) {
  *converged = false;
  const int cap = k + 32;
  const size_t kk = (size_t)k * k, kl = (size_t)k * l;
  T *rows, *X, *Xn, *M, *W, *Y;
  double *nrm, *info;
  JacobiCtl* ctl;
  PrecondStat* stat;
  unsigned char* rbuf;
  SM_CHECK(ctx.scratch("pc.rows", (size_t)cap * k, &rows));
  SM_CHECK(ctx.scratch("pc.nrm", (size_t)cap, &nrm));
  SM_CHECK(ctx.scratch("pc.info", 16, &info));
  SM_CHECK(ctx.scratch("pc.ctl", 1, &ctl));
  SM_CHECK(ctx.scratch("pc.stat", 1, &stat));
  SM_CHECK(ctx.scratch("pc.rbuf", split_cluster_rbuf_bytes(l, k), &rbuf));
  SM_CHECK(ctx.scratch("pc.X", kk, &X));
  SM_CHECK(ctx.scratch("pc.Xn", kk, &Xn));
  SM_CHECK(ctx.scratch("pc.M", kk, &M));
  SM_CHECK(ctx.scratch("pc.W", kl, &W));
  SM_CHECK(ctx.scratch("pc.Y", kl, &Y));
  const T one = S<T>::one(), zero = S<T>::zero();
  PrecondStat* h = reinterpret_cast<PrecondStat*>(ctx.pinned);
  auto read = [&]() -> int {
    SM_CUDA_CHECK(cudaMemcpyAsync(h, stat, sizeof(PrecondStat), cudaMemcpyDeviceToHost, st));
    SM_CUDA_CHECK(cudaStreamSynchronize(st));
    return SM_OK;
  };
  // one Newton-Schulz step; stat->dev and entry: the deviation it started from
  auto newton_schulz = [&]() -> int {
    SM_CUDA_CHECK(cudaMemsetAsync(&stat->dev, 0, 2 * sizeof(double), st));
    SM_CHECK(gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_C, k, k, k, one, X, k, X, k, zero, M, k));
    k_newton_schulz<T><<<k, 128, 0, st>>>(M, k, stat);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
    SM_CHECK(gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_N, k, k, k, one, M, k, X, k, zero, Xn, k));
    std::swap(X, Xn);
    return SM_OK;
  };
  auto angles = [&](double amax) -> int {  // E into M from G in Xn, the verdict into *h
    SM_CUDA_CHECK(cudaMemsetAsync(&stat->einf, 0, sizeof(double) + 2 * sizeof(int), st));
    k_angles<T><<<k, 128, 0, st>>>(Xn, k, l, tol2, use_floor, defl_rel, amax, M, stat);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
    return read();
  };
  // W <- exp(f E) W; f < 1 only where |E|_inf is beyond what kTaylor terms take to
  // rounding (0.05^9 / 9! = 5e-18): the transform stays unitary, the step is shorter
  auto correct = [&](double einf) -> int {
    const double f = einf > kAngleInf ? kAngleInf / einf : 1.0;
    einf *= f;
    int terms = 1;
    double rest = einf * einf / 2.0;  // the first term left out
    while (rest > 1e-17 && terms < kTaylor) {
      ++terms;
      rest *= einf / (terms + 1);
    }
    const T* last = W;
    T* bufs[2] = {Y, rows};  // rows is (k + 32) x k: large enough only for l <= k + 32
    if ((size_t)cap * k < kl) SM_CHECK(ctx.scratch("pc.Y2", kl, &bufs[1]));
    for (int q = terms; q > 1; --q) {
      T* dst = bufs[q & 1];
      SM_CUDA_CHECK(cudaMemcpyAsync(dst, W, sizeof(T) * kl, cudaMemcpyDeviceToDevice, st));
      SM_CHECK(gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_N, k, l, k, S<T>::from_real(f / q), M, k, last,
                           l, one, dst, l));
      last = dst;
    }
    if (last == W) {
      SM_CUDA_CHECK(cudaMemcpyAsync(Y, W, sizeof(T) * kl, cudaMemcpyDeviceToDevice, st));
      last = Y;
    }
    return gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_N, k, l, k, S<T>::from_real(f), M, k, last, l, one, W,
                       l);
  };
  // FP32 stage on `src` (k x l), then W = X src; false in *ok if it gave no basis
  auto level = [&](const T* src, bool* ok) -> int {
    *ok = false;
    SM_CUDA_CHECK(cudaMemsetAsync(ctl, 0, sizeof(JacobiCtl), st));
    SM_CUDA_CHECK(cudaMemsetAsync(stat, 0, sizeof(PrecondStat), st));
    SM_CHECK(split_cluster_f32<T>(st, src, k, l, true, -1.0, 0.0, 40, rows, nrm, cap, ctl, info, 0,
                                  rbuf, false));
    k_rows_to_basis<T><<<cap, 128, 0, st>>>(rows, nrm, cap, k, ctl, X, stat);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
    SM_CHECK(newton_schulz());
    for (int ns = 0; ns < kNewtonSteps; ++ns) {
      SM_CHECK(newton_schulz());
      SM_CHECK(read());
      if (h->status != 0 || h->missing != 0 || !(h->entry <= kDevMax) || !(h->dev <= DBL_MAX))
        return SM_OK;
      if (h->dev <= kDevDone) {
        *ok = true;
        break;
      }
    }
    if (!*ok) return SM_OK;
    return gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_N, k, l, k, one, X, k, src, l, zero,
                       src == W ? Y : W, l);
  };
  bool ok = false;
  SM_CHECK(level(R, &ok));
  if (!ok) return SM_OK;
  int levels = 1;
  for (int s = 0; s < kSteps; ++s) {
    SM_CHECK(gemm_ctx<T>(ctx, st, SM_OP_N, SM_OP_C, k, k, l, one, W, l, W, l, zero, Xn, k));
    SM_CHECK(angles(kAngleMax));
    if (h->viol == 0) {
      *converged = true;
      break;
    }
    const bool rough = h->left > 0 || !(h->einf <= kAngleInf);
    if (rough) SM_CHECK(angles(kAngleSafe));
    SM_CHECK(correct(h->einf));
    if (!rough) continue;
    if (levels == kLevels) break;
    ++levels;
    SM_CHECK(level(W, &ok));
    if (!ok) break;
    std::swap(W, Y);
  }
  SM_CUDA_CHECK(cudaMemcpyAsync(R, W, sizeof(T) * kl, cudaMemcpyDeviceToDevice, st));
  return SM_OK;
}

template bool precondition_takes<double>(Ctx&, int, int);
template bool precondition_takes<cplx>(Ctx&, int, int);
template int precondition_rows<double>(Ctx&, cudaStream_t, double*, int, int, double, int, double,
                                       bool*);
template int precondition_rows<cplx>(Ctx&, cudaStream_t, cplx*, int, int, double, int, double,
                                     bool*);

}  // namespace sm
