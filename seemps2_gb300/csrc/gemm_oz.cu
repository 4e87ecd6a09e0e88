// FP64-accurate GEMM on the BF16 tensor cores (error-free slicing).
//
//   C[M,N] = alpha * op(A)[M,K] * op(B)[K,N] + beta * C      (real, row-major)
//
// GB300 runs FP64 on the CUDA cores only (~1.2 TFLOP/s); its BF16 tensor cores
// run ~2 PFLOP/s dense.  Following the error-free transformation of matrix
// products of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 2012), each
// row of op(A) and each column of op(B) is scaled by a power of two to
// (-1, 1) and cut into S = 8 slices of 7-bit integers,
//   x = 2^(e - 7) * sum_i a_i 2^(-7 i),   a_i in [-127, 127],
// which BF16 holds exactly (stored pre-scaled: a_i 2^(-7 i)).  The product is
//   C = 2^(e_m + e_n - 14) * sum_{i + j <= S - 1} A_i B_j^T
// with the slice products on tcgen05 (kind::f16, BF16 in, FP32 accumulate).
// Each t = i + j has its own FP32 accumulator: over a K chunk of 256,
// sum_{i + j = t} A_i B_j^T is an integer times 2^(-7 t) below
// 4 * 256 * 127^2 < 2^24 for t <= 3, so those four are exact; t = 4..7 (below
// 2^-28 of the leading term) lose at most a bit or two of their own 24.  (The
// tensor cores add an MMA result into an accumulator of a different scale with
// only ~17 bits: one accumulator per scale keeps every addition aligned.)
// After each chunk the exact t = 0..4 (integers in units of 2^(-7 t)) are
// added into one int64 per element (units of 2^-28) and t = 5..7 (below 2^-31
// of the leading term) into an FP32 sum; the two become FP64 once, at the end.
// No FP64 arithmetic runs per chunk (GB300's FP64 pipe would bound it).  The
// truncation after 8 slices (56 bits of each row's range) and the dropped
// products (i + j >= 8) are below 2^-56 of the row / column maxima, so the
// result has the accuracy of an FP64 GEMM.
//
// One CTA (10 warps) per 128 x 64 (128 x 32) output tile and K range:
//   warp 8 / lane 0: TMA, one 3-D box per operand and stage holding all 8
//            slices of a 32-wide K slab (64-byte swizzle), 2 stages;
//   warp 9 / lane 0: 2 x 12 (2 x 8) tcgen05.mma of N = 256 and less, K = 16,
//            per slab into 8 accumulators in TMEM, a commit per stage and per
//            chunk.  (A slice product to an MMA reads A again for each: 4560
//            clocks a slab, shared memory bound, against 2600 and 1800);
//   warps 0-7: per chunk, tcgen05.ld of the 8 accumulators (warp w owns tile
//            rows 32 (w % 4) .. +31, half w / 4 of the columns) into an int64
//            and an FP32 register per element.
// The K ranges of a tile are the CTAs of one cluster.  They leave their int64 and
// FP32 sums in shared memory (where the stages were) and each adds up a share of
// the tile's rows over the cluster and turns it into FP64.  Besides filling the
// SMs, the split divides that conversion, which on a whole 128 x 64 tile takes as
// long as ten slabs' MMAs.  320 x 128 x 256: 14 us after 5 us of preparation; one
// CTA a tile, 64-bit conversions and FP64 partial sums were 30 us after 15 us.
// Every mbarrier wait is bounded; a timeout sets a bit of the status word
// shared with the TF32 path (read by tc_status_check), waits for the CTA's
// copies in flight, frees TMEM and returns.
#include <algorithm>
#include <cfloat>

#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "kernels.cuh"

namespace sm {

namespace cg = cooperative_groups;

namespace {

constexpr int OM = 128, OK = 32, OS = 2;  // tile M, K slab (BF16), stages
constexpr int kSlices = 8;
constexpr int kChunkSlabs = 8;  // 256 of K per exact chunk
constexpr int kGroups = 8;      // one accumulator per t = i + j
constexpr int kOzThreads = 320;  // 8 flush warps, TMA, MMA
constexpr uint32_t kSliceA = OM * OK * 2;  // 8 KB: one slice of A, one slab
// Sizes that follow from the tile's N (64, or 32 where that fills more SMs)
template <int ON>
struct OzTile {
  static constexpr uint32_t kSliceB = ON * OK * 2;
  static constexpr uint32_t kStage = kSlices * (kSliceA + kSliceB);  // 96 KB, 80 KB
  static constexpr size_t kSmem = (size_t)OS * kStage + 1024 + 256;
  static constexpr int kRow = ON + 1;  // row stride of the sums in shared memory: no bank conflicts
  static constexpr uint32_t kCols = kSlices * ON;  // TMEM columns: 8 accumulators
  static constexpr int kGang = 256 / ON;  // slices of B to an MMA
  static_assert((size_t)OM * kRow * 12 <= (size_t)OS * kStage, "the sums fit where the stages were");
};
constexpr int kOzNoExp = -(1 << 28);  // exponent of an all-zero row of an operand
constexpr int kOzNotFinite = 1 << 28;  // and of one with an infinity or a NaN
constexpr int kOzCluster = 8;    // K ranges of a tile that share a cluster (portable size)
// instruction descriptor: D = F32, A = B = BF16, K-major, M = 128
__device__ __forceinline__ constexpr uint32_t oz_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(OM >> 4) << 24);
}
constexpr unsigned long long kOzWaitNs = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, unsigned long long ns) {
  if (mbar_try_wait(b, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (!mbar_try_wait(b, parity))
    if (gtimer() - t0 > ns) return false;
  return true;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                            int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// K-major operand, 64-byte swizzle: rows of 64 B, 8-row atoms of 512 B.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused for this layout)
  d |= (uint64_t)(512 >> 4) << 32;   // stride byte offset
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)4 << 61;            // 64-byte swizzle
  return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t mapa(uint32_t saddr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ long long ld_cluster_s64(uint32_t a) {
  long long v;
  asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// S 2^(e-28) + small 2^e in three FP64 operations: the words of S are the low bits of
// 2^56 (the upper one biased by 2^31, i.e. 2^35 here) and of 2^24, small's bits are
// moved, and 2^e goes onto the exponent's bits unless that leaves the normal range.
// (Every FP64 operation holds the pipe for 64 clocks, a predicated-off one too: what
// is rare is out of line.)
__device__ __noinline__ double oz_outside(double v, int e) {
  return e > kOzNotFinite / 2 ? __hiloint2double(0x7ff80000, 0) : ldexp(v, e);
}
__device__ __noinline__ double oz_axpby(double alpha, double v, double beta, const double* c) {
  return beta == 0.0 ? alpha * v : fma(alpha, v, beta * *c);
}
__device__ __forceinline__ double oz_double(long long S, float small, int e) {
  const int f = __float_as_int(small), x = (f >> 23) & 0xff;
  const double s64 = __hiloint2double(x == 0 ? 0 : (f & 0x80000000) | (x + 896) << 20 | (f & 0x7fffff) >> 3,
                                      x == 0 ? 0 : (int)((unsigned)f << 29));
  const double shi = __hiloint2double(0x43700000, (int)((unsigned long long)S >> 32) ^ 0x80000000);
  const double slo = __hiloint2double(0x41700000, (int)S);
  const double v = ((shi - (72057594037927936.0 + 34359738368.0 + 16777216.0)) + slo) + s64;
  const int hi = __double2hiint(v), xv = (hi >> 20) & 0x7ff;
  if (xv == 0 || xv + e <= 0 || xv + e >= 0x7ff) return oz_outside(v, e);
  return __hiloint2double(hi + (e << 20), __double2loint(v));
}

// Rows r0 .. r1 - 1 of the tile: the sums of the cluster's NZ CTAs in FP64, stored by
// lanes along the columns.  add: C = alpha v + beta C (else C = v)
template <int ON, int NZ>
__device__ __forceinline__ void oz_store(uint32_t base, const int* et, int r0, int r1, int ncol,
                                         bool add, double alpha, double beta, double* C, size_t ldc) {
  uint32_t src[NZ];
#pragma unroll
  for (int y = 0; y < NZ; ++y) src[y] = mapa(base, y);
  const int c = threadIdx.x % ON;
  if (c >= ncol) return;
#pragma unroll 2
  for (int r = r0 + threadIdx.x / ON; r < r1; r += kOzThreads / ON) {
    const uint32_t at = (uint32_t)(r * OzTile<ON>::kRow + c);
    long long S = 0;
    float small = 0.f;
#pragma unroll
    for (int y = 0; y < NZ; ++y) {
      S += ld_cluster_s64(src[y] + at * 8);
      small += ld_cluster_f32(src[y] + (uint32_t)(OM * OzTile<ON>::kRow * 8) + at * 4);
    }
    double v = oz_double(S, small, et[r] + et[OM + c]);
    double* p = C + (size_t)r * ldc + c;
    if (add) v = oz_axpby(alpha, v, beta, p);
    *p = v;
  }
}

template <int ON>
__global__ void __launch_bounds__(kOzThreads, 1)
    k_gemm_oz(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
              const int* __restrict__ ea, const int* __restrict__ eb, int M, int N, int tm,
              int nslabs, int slabs_per, double alpha, double beta, double* __restrict__ C, int ldc,
              double* __restrict__ part, unsigned int* __restrict__ status) {
  using Tile = OzTile<ON>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + (size_t)OS * Tile::kStage);
  uint64_t* empty = full + OS;
  uint64_t* acc_full = empty + OS;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  __shared__ int et[OM + ON];  // exponents of the tile's rows and columns
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // product p: rows p M .. of the slices of A, rows p N .. of those of B (a tile's rows
  // beyond M belong to the next product and are not stored)
  const int p = blockIdx.y / tm, m0 = blockIdx.y % tm * OM, n0 = blockIdx.x * ON;
  if (threadIdx.x < OM) {
    if (m0 + threadIdx.x < M) et[threadIdx.x] = max(ea[p * M + m0 + threadIdx.x], -1100) - 14;
  } else if (threadIdx.x < OM + ON) {
    if (n0 + threadIdx.x - OM < N)
      et[threadIdx.x] = max(eb[p * N + n0 + threadIdx.x - OM], -1100);
  }
  const int s0 = blockIdx.z * slabs_per;
  const int nk = max(0, min(nslabs, s0 + slabs_per) - s0);
  const int nchunks = (nk + kChunkSlabs - 1) / kChunkSlabs;
  if (threadIdx.x == 0) {
    for (int s = 0; s < OS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(Tile::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 8) {
    if (lane == 0) {  // producer
      int issued[OS] = {};
      for (int i = 0; i < nk; ++i) {
        const int s = i % OS;
        const uint32_t ph = (uint32_t)(i / OS) & 1u;
        if (i >= OS && !mbar_wait(&empty[s], ph ^ 1u, kOzWaitNs)) {
          atomicOr(status, 16u);
          break;
        }
        unsigned char* stg = base + (size_t)s * Tile::kStage;
        mbar_expect_tx(&full[s], Tile::kStage);
        const int x = (s0 + i) * OK;
        tma_load_3d(stg, &mA, &full[s], x, p * M + m0, 0);
        tma_load_3d(stg + kSlices * kSliceA, &mB, &full[s], x, p * N + n0, 0);
        issued[s] += 1;
      }
      for (int s = 0; s < OS; ++s)
        if (issued[s] && !mbar_wait(&full[s], (uint32_t)(issued[s] - 1) & 1u, kOzWaitNs))
          atomicOr(status, 64u);
    }
  } else if (warp == 9) {
    if (lane == 0) {  // MMA issuer
      bool failed = false;
      for (int i = 0; i < nk; ++i) {
        const int s = i % OS;
        const uint32_t ph = (uint32_t)(i / OS) & 1u;
        const int c = i / kChunkSlabs, first = (i % kChunkSlabs) == 0;
        // the flush of the previous chunk must have read the accumulators
        if (first && c > 0 && !mbar_wait(acc_empty, (uint32_t)(c - 1) & 1u, kOzWaitNs)) {
          atomicOr(status, 32u);
          failed = true;
          break;
        }
        if (!mbar_wait(&full[s], ph, kOzWaitNs)) {
          atomicOr(status, 32u);
          failed = true;
          break;
        }
        tc_fence_after();
        const uint32_t a0 = smem_u32(base + (size_t)s * Tile::kStage);
        const uint32_t b0 = a0 + kSlices * kSliceA;
        // slice ia of A against slices 0 .. 7 - ia of B, which follow one another in
        // shared memory as their accumulators t = ia .. 7 do in TMEM: up to N = 256
        // to an MMA
#pragma unroll
        for (int kk = 0; kk < OK / 16; ++kk) {
#pragma unroll
          for (int ia = 0; ia < kSlices; ++ia) {
            const uint64_t da = sdesc_sw64(a0 + ia * kSliceA + kk * 32);
#pragma unroll
            for (int jb = 0; jb < kSlices - ia; jb += Tile::kGang) {
              const int n = kSlices - ia - jb < Tile::kGang ? kSlices - ia - jb : Tile::kGang;
              umma_bf16(tmem + (uint32_t)((ia + jb) * ON), da,
                        sdesc_sw64(b0 + jb * Tile::kSliceB + kk * 32), oz_idesc(n * ON),
                        first && kk == 0 && ia == 0 ? 0u : 1u);
            }
          }
        }
        umma_commit(&empty[s]);
        if ((i % kChunkSlabs) == kChunkSlabs - 1 || i == nk - 1) umma_commit(acc_full);
      }
      // after a failed wait the flush still learns when the MMAs issued so far
      // have completed (its next wait then runs out and the CTA returns)
      if (failed) umma_commit(acc_full);
    }
  } else {
    // warps 0-7: per chunk, the exact accumulators t = 0..4 (integers in
    // units of 2^(-7 t)) go into one int64 per element in units of 2^-28;
    // t = 5..7 into an FP32 sum (below 2^-31 of the leading term).  Warp w
    // reads TMEM lanes 32 (w % 4) .. +31 (its lane quadrant), columns
    // 32 (w / 4) .. +31 of each accumulator.
    constexpr int HC = ON / 2;
    const int quad = warp & 3, c0 = (warp >> 2) * HC;
    long long S[HC];
    float small[HC];
#pragma unroll
    for (int j = 0; j < HC; ++j) {
      S[j] = 0;
      small[j] = 0.f;
    }
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      ok = mbar_wait(acc_full, (uint32_t)c & 1u, 4 * kOzWaitNs);
      __syncwarp();
      if (!ok) break;
      tc_fence_after();
      const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
#pragma unroll
      for (int cb = 0; cb < HC; cb += 16) {
        float v[16];
#pragma unroll
        for (int g = 7; g >= 5; --g) {
          tmem_ld16(lane_base + (uint32_t)(g * ON + cb), v);
#pragma unroll
          for (int j = 0; j < 16; ++j) small[cb + j] += v[j];
        }
#pragma unroll
        for (int g = 4; g >= 0; --g) {
          tmem_ld16(lane_base + (uint32_t)(g * ON + cb), v);
          const float up = (float)(1u << (7 * g));  // 2^(7 g): v * up is an integer below 2^25
#pragma unroll
          for (int j = 0; j < 16; ++j)
            S[cb + j] += (long long)__float2int_rn(v[j] * up) << (28 - 7 * g);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
    }
    if (!ok && lane == 0) atomicOr(status, 128u);
    // the last commit has completed: no copy and no MMA uses the stages any more
    long long* Ss = reinterpret_cast<long long*>(base);
    float* Sm = reinterpret_cast<float*>(base + (size_t)OM * Tile::kRow * 8);
    const int at = (quad * 32 + lane) * Tile::kRow + c0;
#pragma unroll
    for (int j = 0; j < HC; ++j) {
      Ss[at + j] = S[j];
      Sm[at + j] = small[j];
    }
  }
  tc_fence_before();
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Tile::kCols)
                 : "memory");
  }
  // this CTA's share of the tile's rows, lanes along the columns
  const int nz = (int)cluster.num_blocks(), z = (int)cluster.block_rank();
  const int mv = min(OM, M - m0), per = (mv + nz - 1) / nz;
  const int r0 = z * per, r1 = min(mv, r0 + per), nc = min(ON, N - n0);
  const uint32_t sums = smem_u32(base);
  const bool add = !part && (alpha != 1.0 || beta != 0.0);
  const size_t ldo = part ? N : ldc;
  double* out = (part ? part + (size_t)(blockIdx.z / nz) * (gridDim.y / tm) * M * N : C) +
                (size_t)(p * M + m0) * ldo + n0;
  switch (nz) {  // a power of two (host)
    case 1: oz_store<ON, 1>(sums, et, r0, r1, nc, add, alpha, beta, out, ldo); break;
    case 2: oz_store<ON, 2>(sums, et, r0, r1, nc, add, alpha, beta, out, ldo); break;
    case 4: oz_store<ON, 4>(sums, et, r0, r1, nc, add, alpha, beta, out, ldo); break;
    default: oz_store<ON, kOzCluster>(sums, et, r0, r1, nc, add, alpha, beta, out, ldo); break;
  }
  cluster.sync();  // no CTA leaves while another reads its sums
}

// One operand of the preparation: op(X) is rows x K with element
// (r, k) = X[r * ldx + k] (trans = 0) or X[k * ldx + r] (trans = 1).  A complex X
// (conjugated if sign is -1) becomes three operands of rows x K, one below the other:
// its real part, its imaginary part, and their sum.
constexpr int kPrepRows = 8;     // rows of a CTA: a warp each
constexpr int kPrepCols = 512;   // K entries held in shared memory
constexpr int kPrepRange = 256;  // K entries of a CTA while the cluster can grow

struct OzOperand {
  const double* X;
  int ldx, rows, trans, sign;
  int* ex;
  __nv_bfloat16* out;
};

// Exponent e (x = f 2^e, f in [0.5, 1)) of the largest |element| of each row of
// op(X) into ex (or kOzNoExp, kOzNotFinite), and the 8 slices of
// op(X) scaled by 2^-ex[r]: out[(i * rows + r) * kp + k] = sign(x) a_i 2^(-7 i)
// (BF16, exact), zero for k >= K, where a_0 a_1 ... a_7 are the base-128 digits of
// |x| 2^-ex[r] < 1, i.e. 7-bit fields of the 56-bit fixed-point value
// F = floor(|x| 2^(56 - ex[r])) taken from the FP64 significand with integer shifts.
//
// A CTA has 8 rows and a K range, a cluster (along y) the whole rows; blockIdx.z
// picks the operand.  The range is read once into shared memory, the maxima go
// through the cluster, and a warp writes the slices of one row, two entries to a
// lane.  Only integer and FP32 operations: maxima of doubles alone, at 64 clocks of
// the FP64 pipe each, took 8 us of the 15 us that separate passes for the exponents
// and the slices did at 320 x 256.
template <int kParts>  // 1: real, 3: complex
__global__ void __launch_bounds__(32 * kPrepRows)
    k_oz_prep(OzOperand A, OzOperand B, int K, int kp, int range) {
  const OzOperand& o = blockIdx.z ? B : A;
  __shared__ __align__(16) double X[kPrepRows][kPrepCols + 2];
  __shared__ unsigned key[kPrepRows];
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rb = gridDim.x / kParts, p = blockIdx.x / rb, r0 = blockIdx.x % rb * kPrepRows;
  if (r0 >= o.rows) return;  // uniform over the cluster
  const int k0 = blockIdx.y * range, k1 = min(kp, k0 + range);
  const int nch = max(1, (k1 - k0 + kPrepCols - 1) / kPrepCols);
  if (tid < kPrepRows) key[tid] = 0;
  __syncthreads();
  // columns c0 .. c0 + n - 1 into X, their maximum (high words; 1 for what is
  // nonzero below them) into key
  auto load = [&](int c0, int n) {
    // trans: 8 rows x 4 columns to a warp, 64 contiguous bytes of each column
    const int rr = o.trans ? tid & 7 : warp, kt = o.trans ? tid >> 3 : lane;
    const bool on = r0 + rr < o.rows;
    constexpr int kWords = kParts == 1 ? 1 : 2;
    const size_t step = (o.trans ? (size_t)o.ldx : 1) * kWords;
    const double* src =
        o.X + (o.trans ? (size_t)(r0 + rr) : (size_t)(r0 + rr) * o.ldx) * kWords + c0 * step;
    unsigned m = 0;
    for (int ka = kt; ka < n; ka += 8 * 32) {  // eight loads in flight
      double x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = ka + 32 * i;
        x[i] = 0.0;
        if (on && k < n && c0 + k < K) {
          if (kParts == 1 || p == 0) x[i] = src[k * step];
          else if (p == 1) x[i] = o.sign < 0 ? -src[k * step + 1] : src[k * step + 1];
          else x[i] = o.sign < 0 ? src[k * step] - src[k * step + 1] : src[k * step] + src[k * step + 1];
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = ka + 32 * i;
        if (k < n) X[rr][k] = x[i];
        m = max(m, (unsigned)(__double2hiint(x[i]) & 0x7fffffff) | (__double2loint(x[i]) != 0));
      }
    }
    if (o.trans) {
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
      if (lane < 8) atomicMax(&key[rr], m);
    } else {
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) atomicMax(&key[rr], m);
    }
  };
  for (int c = 0; c < nch; ++c) {
    if (c) __syncthreads();
    load(k0 + c * kPrepCols, min(kPrepCols, k1 - k0 - c * kPrepCols));
  }
  cluster.sync();
  const int r = r0 + warp;
  unsigned m = 0;
  for (int y = 0; y < (int)cluster.num_blocks(); ++y)
    m = max(m, *cluster.map_shared_rank(&key[warp], y));
  // the bound 2^-1021 of a row of subnormals loses none of their bits
  const int ex = m == 0 ? kOzNoExp
                        : m >= 0x7ff00000u ? kOzNotFinite : max((int)(m >> 20), 1) - 1022;
  if (cluster.block_rank() == 0 && lane == 0 && r < o.rows) o.ex[p * o.rows + r] = ex;
  const size_t plane = (size_t)kParts * o.rows * kp;
  __nv_bfloat16* out = o.out + (size_t)(p * o.rows + r) * kp;
  for (int c = 0; c < nch; ++c) {
    const int c0 = k0 + c * kPrepCols, n = min(kPrepCols, k1 - c0);
    if (nch > 1) {
      __syncthreads();
      load(c0, n);
      __syncthreads();
    }
    if (r >= o.rows) continue;
    for (int k = 2 * lane; k < n; k += 64) {
      unsigned long long F[2];
      unsigned sign[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned long long bits = (unsigned long long)__double_as_longlong(X[warp][k + h]);
        const int bexp = (int)((bits >> 52) & 0x7FF);
        // |x| = f 2^(ev - 52) < 2^ex, so the shift is at most 3
        const unsigned long long f = (bits & ((1ull << 52) - 1)) | (bexp ? 1ull << 52 : 0ull);
        const int sh = (bexp ? bexp - 1023 : -1022) - ex + 4;
        F[h] = f == 0 ? 0ull : sh >= 0 ? f << (sh & 63) : (sh > -64 ? f >> (-sh) : 0ull);
        sign[h] = (unsigned)(bits >> 32) & 0x80000000u;
      }
      float scale = 1.f;
#pragma unroll
      for (int i = 0; i < kSlices; ++i) {
        unsigned w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // the digit as a float: 2^23 + a - 2^23
          const unsigned a = (unsigned)(F[h] >> (49 - 7 * i)) & 127u;
          w[h] = __float_as_uint((__uint_as_float(0x4B000000u | a) - 8388608.0f) * scale) | sign[h];
        }
        *reinterpret_cast<unsigned*>(out + i * plane + c0 + k) =
            __byte_perm(w[0], w[1], 0x7632);
        scale *= 0.0078125f;  // 2^-7
      }
    }
  }
  cluster.sync();  // no CTA leaves while another reads its maxima
}

// C = alpha sum_z part_z + beta C: the clusters of one tile
__global__ void k_oz_reduce(int M, int N, int nz, const double* __restrict__ part, double alpha,
                            double beta, double* __restrict__ C, int ldc) {
  const size_t mn = (size_t)M * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < mn;
       e += (size_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int z = 0; z < nz; ++z) acc += part[(size_t)z * mn + e];
    double* p = C + (e / N) * ldc + (e % N);
    *p = beta == 0.0 ? alpha * acc : fma(alpha, acc, beta * *p);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 oz_encode_fn() {
  // looked up once (thread-safe static initialisation); null when unavailable
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    cudaGetLastError();
    return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
  }();
  return fn;
}

// 3-D map over the slices: (k, row, slice), box (32, box_rows, 8), 64-byte swizzle
int make_slice_map(CUtensorMap* map, const __nv_bfloat16* base, int rows, int kp, int box_rows) {
  auto enc = oz_encode_fn();
  if (!enc) {
    set_error("FP64 tensor-core GEMM: cuTensorMapEncodeTiled not available");
    return SM_ERR_CUDA;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)kSlices};
  const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)rows * kp * 2};
  const cuuint32_t box[3] = {(cuuint32_t)OK, (cuuint32_t)box_rows, (cuuint32_t)kSlices};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                         const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("FP64 tensor-core GEMM: tensor map encoding failed");
    return SM_ERR_CUDA;
  }
  return SM_OK;
}

}  // namespace

namespace {

template <typename... P, typename... Q>
int cluster_launch(void (*fn)(P...), dim3 grid, dim3 block, dim3 cluster, size_t smem,
                   cudaStream_t st, Q... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster.x;
  attr.val.clusterDim.y = cluster.y;
  attr.val.clusterDim.z = cluster.z;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  SM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fn, args...));
  return SM_OK;
}

}  // namespace

bool gemm_oz_eligible(int M, int N, int K) {
  return (double)M * N * K >= 2.0 * 1024 * 1024 && M >= 32 && N >= 32 && K >= 32 &&
         oz_encode_fn() != nullptr;
}

namespace {

// parts products of M x N x K, the p-th at rows p M .. of C
template <int kParts>
int products(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, double alpha,
             const double* A, int lda, const double* B, int ldb, double beta, double* C, int ldc) {
  const int kp = (K + OK - 1) / OK * OK;
  const int nslabs = kp / OK;
  __nv_bfloat16 *sa, *sb;
  int *ea, *eb;
  unsigned int* status;
  SM_CHECK(ctx.scratch("oz.A", (size_t)kSlices * kParts * M * kp, &sa));
  SM_CHECK(ctx.scratch("oz.B", (size_t)kSlices * kParts * N * kp, &sb));
  SM_CHECK(ctx.scratch("oz.ea", (size_t)kParts * M, &ea));
  SM_CHECK(ctx.scratch("oz.eb", (size_t)kParts * N, &eb));
  SM_CHECK(tc_status(ctx, &status));
  // op(A)[m][k] = A[m][k] (N) or A[k][m] (T, C: real); op(B)^T[n][k] = B[k][n]
  // (N) or B[n][k] (T, C)
  const int ta = opA == SM_OP_N ? 0 : 1, tb = opB == SM_OP_N ? 1 : 0;
  const OzOperand oa{A, lda, M, ta, opA == SM_OP_C ? -1 : 1, ea, sa};
  const OzOperand ob{B, ldb, N, tb, opB == SM_OP_C ? -1 : 1, eb, sb};
  const int rb = (std::max(M, N) + kPrepRows - 1) / kPrepRows;
  const int zk = std::min(kOzCluster, (kp + kPrepRange - 1) / kPrepRange);
  const int range = (nslabs + zk - 1) / zk * OK;
  SM_CHECK(cluster_launch(k_oz_prep<kParts>, dim3(kParts * rb, zk, 2), dim3(32 * kPrepRows), dim3(1, zk, 1), 0, st,
                          oa, ob, K, kp, range));
  note_launch();
  CUtensorMap mA, mB;
  SM_CHECK(make_slice_map(&mA, sa, kParts * M, kp, OM));
  // Split K over the CTAs of a cluster while the output has fewer tiles than SMs,
  // down to one slab each (any split at slabs is exact).  Only beyond 16 slabs a CTA
  // a tile gets several clusters: their sum is another launch of ~4 us.
  const int sms = std::max(1, ctx.num_sms), tm = (M + OM - 1) / OM;
  const int tiles = kParts * tm * ((N + 63) / 64);
  SM_CHECK(raise_smem_limit(k_gemm_oz<64>, OzTile<64>::kSmem));
  int nmax = kOzCluster;  // the largest cluster that finds room, at one CTA to an SM in either width
  while (nmax > 1 && !ctx.places(reinterpret_cast<const void*>(k_gemm_oz<64>), nmax, kOzThreads,
                                 OzTile<64>::kSmem))
    nmax /= 2;
  int nz = 1;
  while (nz < nmax && 2 * nz <= std::min(sms / tiles, nslabs)) nz *= 2;
  int slabs_per = (nslabs + nz - 1) / nz;
  const int nzo =
      nz < nmax ? 1 : std::max(1, std::min(sms / (tiles * nz), slabs_per / 8));
  if (nzo > 1) slabs_per = (nslabs + nz * nzo - 1) / (nz * nzo);
  double* part = nullptr;
  if (nzo > 1) SM_CHECK(ctx.scratch("oz.part", (size_t)nzo * kParts * M * N, &part));
  // Half as wide a tile where twice as many CTAs still find an SM each: half of
  // everything but the loads of A to a CTA.
  const bool narrow = 2 * tiles * nz * nzo <= sms && N > 32;
  const int on = narrow ? 32 : 64;
  SM_CHECK(make_slice_map(&mB, sb, kParts * N, kp, on));
  const auto kernel = narrow ? k_gemm_oz<32> : k_gemm_oz<64>;
  const size_t smem = narrow ? OzTile<32>::kSmem : OzTile<64>::kSmem;
  SM_CHECK(raise_smem_limit(kernel, smem));
  SM_CHECK(cluster_launch(kernel, dim3((N + on - 1) / on, kParts * tm, nz * nzo), dim3(kOzThreads),
                          dim3(1, 1, nz), smem, st, mA, mB, (const int*)ea, (const int*)eb, M, N, tm,
                          nslabs, slabs_per, alpha, beta, C, ldc, part, status));
  note_launch();
  if (nzo > 1) {
    const size_t mn = (size_t)kParts * M * N;
    k_oz_reduce<<<(int)std::min<size_t>((mn + 255) / 256, 4096), 256, 0, st>>>(kParts * M, N, nzo, part,
                                                                               alpha, beta, C, ldc);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
  }
  return SM_OK;
}

}  // namespace

int gemm_oz(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, double alpha,
            const double* A, int lda, const double* B, int ldb, double beta, double* C, int ldc) {
  return products<1>(ctx, st, opA, opB, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
}

int gemm_oz_3m(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, const cplx* A,
               int lda, const cplx* B, int ldb, double* T) {
  return products<3>(ctx, st, opA, opB, M, N, K, 1.0, &A->re, lda, &B->re, ldb, 0.0, T, N);
}

}  // namespace sm
