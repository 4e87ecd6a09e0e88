// One Lanczos run on the two-site operator (dmrg.cu), its scalars kept on the device.
//
// Step j: w = H V[j]; the overlaps of w with all vectors so far are taken out twice
// (classical Gram-Schmidt, FP64), alpha_j is the first pass's own, beta_j = |w|, and
// V[j + 1] = w / beta_j.  The reference calls ARPACK for this (optimization/dmrg.py:
// 15-23).  The kernels store the alphas and betas in host memory too, and before the host
// issues a step it looks at the one two before: a run that breaks down (an invariant
// subspace: a start that is an eigenvector, a small block) ends there, with one
// unused step issued, and the device has a step to do while the host issues the next.  A step is the matvec
// and five kernels; with a dozen calls from Python and two reads of a scalar per step,
// 30 steps at bond 108 took 160 us a step beyond the matvec's kernels.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace sm {

namespace {

constexpr int kChunk = 512;   // vector elements per block of the overlaps
constexpr int kLanNT = 256;
constexpr double kBreakdown = 1e-14;  // beta of an invariant subspace, relative to the alphas
constexpr int kLead = 2;          // a step is issued once the beta of the kLead-th before it is seen
constexpr size_t kLanPinned = 60 * 1024;  // their alphas and betas in the pinned block (bytes)

// Overlaps coef[i] = V[i] . w, i < rows: block b holds one chunk of w in shared
// memory, warp k takes rows k, k + 8, ..; the last block to finish adds the blocks'
// parts in order and stores coef[rows - 1] to *alpha and *host too (if given).  A lane adds 16
// products before the warp's five shuffle sums: each FP64 instruction costs its warp
// 64 clocks whether it adds products or partial sums.
__global__ void __launch_bounds__(kLanNT) k_lan_dots(const double* __restrict__ V, int rows, int n,
                                                     const double* __restrict__ w,
                                                     double* __restrict__ part,
                                                     double* __restrict__ coef, double* alpha,
                                                     double* host, unsigned int* done) {
  __shared__ double ws[kChunk];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * kChunk, nx = min(kChunk, n - x0);
  for (int x = threadIdx.x; x < nx; x += kLanNT) ws[x] = w[x0 + x];
  __syncthreads();
  for (int i = warp; i < rows; i += kLanNT / 32) {
    const double* v = V + (size_t)i * n + x0;
    double a = 0.0;
    for (int x = lane; x < nx; x += 32) a = fma(v[x], ws[x], a);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) __stcg(part + (size_t)i * gridDim.x + blockIdx.x, a);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = warp; i < rows; i += kLanNT / 32) {
    double a = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) a += __ldcg(part + (size_t)i * gridDim.x + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) {
      coef[i] = a;
      if (alpha && i == rows - 1) *alpha = *host = a;
    }
  }
  if (threadIdx.x == 0) *done = 0u;
}

// w -= sum_i coef[i] V[i]; with `beta`, also *beta = *host = |w| (the last block adds the
// blocks' sums of squares in order).
__global__ void __launch_bounds__(kLanNT) k_lan_update(const double* __restrict__ V, int rows, int n,
                                                       const double* __restrict__ coef,
                                                       double* __restrict__ w, double* __restrict__ part,
                                                       double* beta, double* host,
                                                       unsigned int* done) {
  __shared__ double red[kLanNT / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = blockIdx.x * kLanNT + threadIdx.x;
  double v = 0.0;
  if (x < n) {
    double a0 = 0.0, a1 = 0.0;
    int i = 0;
    for (; i + 1 < rows; i += 2) {
      a0 = fma(coef[i], V[(size_t)i * n + x], a0);
      a1 = fma(coef[i + 1], V[(size_t)(i + 1) * n + x], a1);
    }
    if (i < rows) a0 = fma(coef[i], V[(size_t)i * n + x], a0);
    v = w[x] - (a0 + a1);
    w[x] = v;
  }
  if (!beta) return;
  double s = v * v;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < kLanNT / 32; ++k) t += red[k];
    __stcg(part + blockIdx.x, t);
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || warp != 0) return;
  __threadfence();
  double t = 0.0;
  for (int b = lane; b < (int)gridDim.x; b += 32) t += __ldcg(part + b);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) {
    *beta = *host = sqrt(t);
    *done = 0u;
  }
}

// y = x / *norm (zero if the norm is not positive)
__global__ void k_lan_scale(const double* __restrict__ x, int n, const double* __restrict__ norm,
                            double* __restrict__ y) {
  const double b = *norm, r = b > 0.0 ? 1.0 / b : 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = r * x[i];
}

}  // namespace

int lanczos_run(Ctx& ctx, cudaStream_t st, const int* d, const double* L, const double* H,
                const double* R, int precision, bool prepared, const double* x0, int m, double* V,
                double* alpha, double* beta, int* steps) {
  const size_t n64 = (size_t)d[2] * d[3] * d[4] * d[7];
  if (n64 != (size_t)d[0] * d[3] * d[4] * d[6] || n64 > 0x7fffffff) {
    set_error("lanczos: the operator must be square");
    return SM_ERR_VALUE;
  }
  if (prepared) {  // its matvec goes by its own sizes and environments
    const MatvecPrep& mp = ctx.mvp;
    const int own[8] = {mp.a, mp.c, mp.b, mp.p1, mp.p2, mp.e, mp.g, mp.f};
    if (mp.precision != precision || mp.L != L || mp.R != R || !std::equal(own, own + 8, d)) {
      set_error("lanczos: the context holds another prepared operator (sm_two_site_prepare)");
      return SM_ERR_VALUE;
    }
  }
  const int n = (int)n64;
  m = std::max(1, std::min(m, n));
  const int nb = (n + kChunk - 1) / kChunk, ub = (n + kLanNT - 1) / kLanNT;
  double *w, *part, *coef, *ab;
  unsigned int* done;
  SM_CHECK(ctx.scratch("lan.w", (size_t)n, &w));
  SM_CHECK(ctx.scratch("lan.part", std::max((size_t)m * nb, (size_t)ub), &part));
  SM_CHECK(ctx.scratch("lan.coef", (size_t)m, &coef));
  SM_CHECK(ctx.scratch("lan.ab", 2 * (size_t)m + 1, &ab));  // alphas, betas, |x0|
  SM_CHECK(ctx.scratch("lan.done", 1, &done));
  SM_CUDA_CHECK(cudaMemsetAsync(done, 0, sizeof(unsigned int), st));
  const int sb = std::min(ub, 1024);
  for (cudaEvent_t& e : ctx.lan)
    if (!e) SM_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  // [step % kLead][alpha, beta], and |x0|
  volatile double* seen = reinterpret_cast<double*>(static_cast<char*>(ctx.pinned) + kLanPinned);
  double* seen_dev = const_cast<double*>(seen);
  int run = 0;  // steps issued
  double largest = 0.0;
  // V[0] = x0 / |x0|: no vectors to take out, the norm alone
  SM_CUDA_CHECK(cudaMemcpyAsync(w, x0, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  k_lan_update<<<ub, kLanNT, 0, st>>>(V, 0, n, coef, w, part, ab + 2 * m,
                                      seen_dev + 2 * kLead, done);
  k_lan_scale<<<sb, kLanNT, 0, st>>>(w, n, ab + 2 * m, V);
  note_launch(2);
  for (int j = 0; j < m; ++j) {
    double* slot = seen_dev + 2 * (j % kLead);
    if (j >= kLead) {
      SM_CUDA_CHECK(cudaEventSynchronize(ctx.lan[j % kLead]));
      largest = std::max(largest, std::fabs(seen[2 * (j % kLead)]));
      if (seen[2 * (j % kLead) + 1] <= kBreakdown * largest) break;
    }
    run = j + 1;
    const double* q = V + (size_t)j * n;
    if (prepared) SM_CHECK(two_site_matvec_prepared(ctx, st, H, q, w));
    else
      SM_CHECK(two_site_matvec<double>(ctx, st, d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], L, H, R,
                                       q, w, precision));
    for (int pass = 0; pass < 2; ++pass) {
      k_lan_dots<<<nb, kLanNT, 0, st>>>(V, j + 1, n, w, part, coef, pass ? nullptr : ab + j, slot,
                                        done);
      k_lan_update<<<ub, kLanNT, 0, st>>>(V, j + 1, n, coef, w, part, pass ? ab + m + j : nullptr,
                                          slot + 1, done);
    }
    note_launch(4);
    SM_CUDA_CHECK(cudaEventRecord(ctx.lan[j % kLead], st));
    if (j + 1 < m) {
      k_lan_scale<<<sb, kLanNT, 0, st>>>(w, n, ab + m + j, V + (size_t)(j + 1) * n);
      note_launch();
    }
  }
  SM_CUDA_CHECK(cudaGetLastError());
  std::vector<double> h(2 * (size_t)m + 1);
  SM_CUDA_CHECK(cudaMemcpyAsync(h.data(), ab, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st));
  SM_CUDA_CHECK(cudaStreamSynchronize(st));
  if (h[2 * m] == 0.0) {
    set_error("lanczos: the start vector is zero");
    return SM_ERR_VALUE;
  }
  if (prepared || precision != SM_MATVEC_FP64) SM_CHECK(tc_status_check(ctx, st));
  double amax = 0.0;
  for (int j = 0; j < run; ++j) {
    alpha[j] = h[j];
    beta[j] = h[m + j];
    *steps = j + 1;
    amax = std::max(amax, std::fabs(h[j]));
    if (beta[j] <= kBreakdown * amax) break;  // an invariant subspace: the Ritz pair is exact
  }
  return SM_OK;
}

}  // namespace sm
