// What the two kernels of the FP32 stage (svd_cluster_qr.cu, svd_cluster_jacobi.cu)
// share: FP32 element helpers, packed FP32 pairs, mbarriers and stores to other CTAs
// of the cluster.
#pragma once

#include <cfloat>
#include <cstdint>

#include "kernels.cuh"

namespace sm {

constexpr int kCNT = 512;          // threads per CTA
constexpr int kCNW = kCNT / 32;    // warps per CTA
constexpr int kCWMax = 16;         // CTAs per cluster at most
constexpr int kMaxRows = 512;      // rows of R at most (16 CTAs, two blocks of <= 16 rows each)
constexpr int kMaxCol = 1024;      // rows of W at most
constexpr unsigned long long kClusterWaitNs = 1000000000ull;  // 1 s per wait

// ---- FP32 element helpers ----------------------------------------------------
template <typename T> struct F32;
template <> struct F32<double> {
  using type = float;
  __device__ static float from(double x, double s) { return (float)(x * s); }
  __device__ static double to(float x, double s) { return (double)x * s; }
  __device__ static float zero() { return 0.0f; }
};
template <> struct F32<cplx> {
  using type = float2;
  __device__ static float2 from(cplx x, double s) {
    return make_float2((float)(x.re * s), (float)(x.im * s));
  }
  __device__ static cplx to(float2 x, double s) { return cplx{(double)x.x * s, (double)x.y * s}; }
  __device__ static float2 zero() { return make_float2(0.f, 0.f); }
};

__device__ __forceinline__ float f_abs2(float x) { return x * x; }
__device__ __forceinline__ float f_abs2(float2 x) { return fmaf(x.x, x.x, x.y * x.y); }
// acc += conj(u) v
__device__ __forceinline__ void f_dotc(float u, float v, float& gr, float&) { gr = fmaf(u, v, gr); }
__device__ __forceinline__ void f_dotc(float2 u, float2 v, float& gr, float& gi) {
  gr = fmaf(u.x, v.x, fmaf(u.y, v.y, gr));
  gi = fmaf(u.x, v.y, fmaf(-u.y, v.x, gi));
}
// c -= (wr + i wi) v
__device__ __forceinline__ void f_axpy(float wr, float, float v, float& c) { c = fmaf(-wr, v, c); }
__device__ __forceinline__ void f_axpy(float wr, float wi, float2 v, float2& c) {
  c.x = fmaf(-wr, v.x, fmaf(wi, v.y, c.x));
  c.y = fmaf(-wr, v.y, fmaf(-wi, v.x, c.y));
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// the SFU's reciprocal root and reciprocal (a few ulp; arguments well inside the range)
__device__ __forceinline__ float f_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float f_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---- packed FP32 pairs (one instruction for two lanes of a 64-bit register) ----
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
  f2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
  f2_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
  f2_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
  f2_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float f2_hsum(f2_t v) {
  float lo, hi;
  f2_unpack(v, lo, hi);
  return lo + hi;
}
// (x, y) -> (y, -x): the complex number times -i
__device__ __forceinline__ f2_t f2_mul_mi(f2_t v) {
  float x, y;
  f2_unpack(v, x, y);
  return f2_pack(y, -x);
}

// ---- mbarriers and stores across the cluster -----------------------------------
__device__ __forceinline__ uint32_t cl_smem(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cl_map(uint32_t addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(cl_smem(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void cl_mbar_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void cl_mbar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cl_smem(b)), "r"(bytes)
               : "memory");
}
// one arrival on an mbarrier of any CTA of the cluster (a cl_map'ed address)
__device__ __forceinline__ void cl_mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool cl_mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(cl_smem(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// waits for the phase of the given parity; false after kClusterWaitNs
__device__ __forceinline__ bool cl_mbar_wait(uint64_t* b, uint32_t parity) {
  if (cl_mbar_try(b, parity)) return true;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  while (!cl_mbar_try(b, parity)) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > kClusterWaitNs) return false;
  }
  return true;
}
// this CTA's shared memory by its 32-bit address (pointers that vary in a loop become
// generic loads: 64-bit address arithmetic and a longer way)
__device__ __forceinline__ void cl_lds16(uint32_t addr, f2_t& a, f2_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ void cl_sts16(uint32_t addr, f2_t a, f2_t b) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ float cl_lds(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cl_sts(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// `bytes` (a multiple of 16) from this CTA's shared memory into another's, counted by
// that CTA's mbarrier; the source was written with cl_bulk_fence after it
__device__ __forceinline__ void cl_bulk(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst),
      "r"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void cl_bulk_fence() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// shared-memory limit and cluster size of a kernel of the stage
template <typename K>
int cl_allow(K* fn, size_t smem) {
  SM_CHECK(raise_smem_limit(fn, smem));
  SM_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return SM_OK;
}
// one cluster of nc CTAs
template <typename... P, typename... Q>
int cl_launch(void (*fn)(P...), int nc, size_t smem, cudaStream_t st, Q... args) {
  SM_CHECK(cl_allow(fn, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nc);
  cfg.blockDim = dim3(kCNT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = nc;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  SM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fn, args...));
  note_launch();
  return SM_OK;
}
template <typename K>
bool cl_places(Ctx& ctx, K* fn, int nc, size_t smem) {
  return cl_allow(fn, smem) == SM_OK && ctx.places(reinterpret_cast<const void*>(fn), nc, kCNT, smem);
}

// ---- between the two kernels ---------------------------------------------------
// Rows of R padded to whole 16-byte vectors of 32 lanes: R is column-major with
// this column stride.  0: beyond the kernels' sizes.
template <typename T>
int qr_row_pad(int kw);
template <typename T>
bool qr_cluster_ok(Ctx& ctx, int kw, int l);
// Rank-revealing Householder QR of W = (trans ? A^T : A) (kw x l) / |W|_F: R into Rg,
// ctl->nact = its rows, ctl->plateau = 1 if it stopped at the FP32 noise level,
// info[0] = |W|_F^2 (FP64), info[1] the weight below the rows.
template <typename T>
int qr_cluster(cudaStream_t st, const T* A, int n_a, int trans, int kw, int l, double thr_rel,
               double thr_abs, typename F32<T>::type* Rg, JacobiCtl* ctl, double* info, int qr_cap,
               const int* cap_dev, int pivot, int plateau);
// One-sided Jacobi on the ctl->nact (<= kmax) rows of R (length l): kcap rows (FP64,
// times sqrt(info[0])) and their norms.
template <typename T>
bool jacobi_cluster_ok(Ctx& ctx, int kmax, int l);
template <typename T>
int jacobi_cluster(cudaStream_t st, const typename F32<T>::type* Rg, int ldk, int kmax, int l,
                   int max_sweeps, T* out_rows, double* out_nrm, int kcap, JacobiCtl* ctl,
                   double* info);

}  // namespace sm
