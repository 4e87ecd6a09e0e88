// Tensor-core GEMM for FP64 operands at FP32 accuracy: 3xTF32 on tcgen05.
//
//   C[M,N] = alpha * op(A)[M,K] * op(B)[K,N] + beta * C      (real, row-major)
//
// The mixed precision forms run the sweep contractions (cython/gemm.pxi:21-122
// in the reference, FP64 there) at FP32 accuracy.  GB300's CUDA cores give
// FP32 at 64x the FP64 rate, its tensor cores TF32 at another ~15x; TF32 keeps
// 11 significant bits, so each operand is split x = hi + lo (hi = x rounded to
// TF32, lo = the FP32 rest) and the product is hi*hi + hi*lo + lo*hi
// accumulated in FP32 in tensor memory: the error of an FP32 GEMM.
//
// Data path per 128 x 128 output tile (one CTA of 128 threads and K range; the K ranges
// of a tile are the CTAs of a cluster, taken when the output has few tiles):
//   * a split kernel writes hi / lo of op(A) as M x Kp and of op(B)^T as
//     N x Kp FP32 arrays (K contiguous, Kp = K rounded up to 32, zero pad);
//   * warp 0 / lane 0 streams 32-wide K slices of the four arrays with TMA
//     (cp.async.bulk.tensor, 128-byte swizzle) into a 3-stage ring;
//   * warp 1 / lane 0 issues tcgen05.mma kind::tf32 (M=128, N=128, K=8; three
//     per K step) into 4 accumulators of 128 TMEM columns in turn, and
//     tcgen05.commit frees each stage;
//   * all four warps read the accumulators back with tcgen05.ld (warp w owns
//     TMEM lanes 32w..32w+31 = tile rows), leave their sum in shared memory, and
//     each CTA adds up a share of the rows over the cluster and stores it.
// 320 x 128 x 256 takes 10 us after 6 us of splitting.  (Planes in a launch for each
// operand, an epilogue that widened and stored a row to a lane, FP64 partial sums in
// memory and a pass over them: 15, 12 and 4.5 us.)
// Every mbarrier wait is bounded (globaltimer): on timeout the CTA records an
// error bit, waits (bounded) for its own copies in flight, frees its TMEM and
// returns; the sweep reads the status word at its end.
#include <algorithm>

#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "kernels.cuh"

namespace sm {

namespace cg = cooperative_groups;

namespace {

constexpr int TM = 128, TN = 128, TS = 3;
constexpr int kTCThreads = 128;
constexpr int kTcCluster = 8;   // K ranges of a tile that share a cluster (portable size)
constexpr int kTcRow = TN + 1;  // row stride of the sums in shared memory: no bank conflicts
// Per mode: 3xTF32 (FP32 planes hi and lo of both operands, 32-wide K slabs,
// three tf32 MMAs of K = 8 per 8 of K) or BF16 (one BF16 plane per operand,
// 64-wide K slabs, one f16-kind MMA of K = 16 per 16 of K).  Either way a
// slab row is 128 bytes, the span of the 128-byte swizzle.
template <bool BF16>
struct TcMode {
  static constexpr int TK = BF16 ? 64 : 32;          // K elements per slab
  static constexpr int KMMA = BF16 ? 16 : 8;         // K per MMA instruction
  static constexpr int planes = BF16 ? 1 : 2;        // planes per operand
  static constexpr uint32_t tileA = TM * 128;        // bytes of one plane's slab
  static constexpr uint32_t tileB = TN * 128;
  static constexpr uint32_t stage = planes * (tileA + tileB);
  static constexpr size_t smem = (size_t)TS * stage + 1024 + 256;
  // accumulators that the slabs take turns in
  static constexpr int acc = BF16 ? 1 : 4;
  // instruction descriptor: D = F32 (bits 4-5 = 1), A and B TF32 (2) or BF16
  // (1) at bits 7-9 and 10-12, both K-major (bits 15, 16 = 0), N >> 3 at bits
  // 17-22, M >> 4 at bits 24-28
  static constexpr uint32_t fmt = BF16 ? 1u : 2u;
  static constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) |
                                    ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
};
static_assert((size_t)TM * kTcRow * 4 <= (size_t)TS * TcMode<true>::stage,
              "the sums fit where the stages were");
constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s per wait

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
// Waits for the phase of the given parity; false after `ns` nanoseconds.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, unsigned long long ns) {
  if (mbar_try_wait(b, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (!mbar_try_wait(b, parity))
    if (gtimer() - t0 > ns) return false;
  return true;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                            int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, "
      "%4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// K-major operand in the 128-byte swizzled layout TMA writes: rows of 128 B,
// 8-row atoms of 1024 B (stride byte offset), descriptor version 1.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;              // leading byte offset (unused for this layout)
  d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;              // descriptor version
  d |= (uint64_t)2 << 61;              // 128-byte swizzle
  return d;
}
__device__ __forceinline__ void umma_tf32(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(TcMode<false>::idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(TcMode<true>::idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane
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
__device__ __forceinline__ float ld_cluster_f32(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
// FP32 to FP64 by integer operations: a conversion holds the FP64 pipe for 64 clocks, a
// predicated-off one too, so what is rare (subnormal, infinite, NaN) is out of line
__device__ __noinline__ double tc_widen_rare(float f) { return (double)f; }
__device__ __forceinline__ double tc_widen(float f) {
  const unsigned b = __float_as_uint(f), x = (b >> 23) & 0xffu;
  if ((b << 1) != 0 && (x == 0 || x == 0xffu)) return tc_widen_rare(f);
  const unsigned hi = (b << 1) == 0 ? b : (b & 0x80000000u) | ((x + 896u) << 20) | ((b & 0x7fffffu) >> 3);
  return __hiloint2double((int)hi, (int)((b << 1) == 0 ? 0u : b << 29));
}
template <typename OutT>
__device__ __noinline__ void tc_axpby(double alpha, double v, double beta, OutT* c) {
  *c = beta == 0.0 ? (OutT)(alpha * v) : (OutT)fma(alpha, v, beta * (double)*c);
}

// Rows r0 .. r1 - 1 of the tile: the sum of the cluster's NZ FP32 tiles, carried as an
// unevaluated sum of two FP32 (48 bits) so that FP64 adds once, stored by lanes along
// the columns.  add: C = alpha v + beta C (else C = v)
template <int NZ, typename OutT>
__device__ __forceinline__ void tc_store(uint32_t base, int r0, int r1, int ncol, bool add,
                                         double alpha, double beta, OutT* C, size_t ldc) {
  uint32_t src[NZ];
#pragma unroll
  for (int y = 0; y < NZ; ++y) src[y] = mapa(base, y) + threadIdx.x * 4;
  const int c = threadIdx.x;  // kTCThreads == TN
  if (c >= ncol) return;
#pragma unroll 4
  for (int r = r0; r < r1; ++r) {
    float hi = ld_cluster_f32(src[0] + (uint32_t)(r * kTcRow * 4)), lo = 0.f;
#pragma unroll
    for (int y = 1; y < NZ; ++y) {
      const float x = ld_cluster_f32(src[y] + (uint32_t)(r * kTcRow * 4));
      const float t = hi + x, u = t - hi;
      lo += (hi - (t - u)) + (x - u);
      hi = t;
    }
    OutT* p = C + (size_t)r * ldc + c;
    if (NZ > 1 && !(fabsf(lo) <= FLT_MAX)) lo = 0.f;  // an infinity in hi stays one
    if (add) {
      tc_axpby<OutT>(alpha, (double)hi + (double)lo, beta, p);
    } else if constexpr (sizeof(OutT) == 8) {
      *p = NZ > 1 ? tc_widen(hi) + tc_widen(lo) : tc_widen(hi);
    } else {
      *p = hi + lo;
    }
  }
}

template <bool BF16, typename OutT>
__global__ void __launch_bounds__(kTCThreads, 1)
    k_gemm_tc(const __grid_constant__ CUtensorMap mAh, const __grid_constant__ CUtensorMap mAl,
              const __grid_constant__ CUtensorMap mBh, const __grid_constant__ CUtensorMap mBl,
              int M, int N, int ktiles, int kt_per, double alpha, double beta,
              OutT* __restrict__ C, int ldc, OutT* __restrict__ part,
              unsigned int* __restrict__ status) {
  using Md = TcMode<BF16>;
  constexpr uint32_t kStage = Md::stage, kTileA = Md::tileA, kTileB = Md::tileB;
  constexpr int TK = Md::TK;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + (size_t)TS * kStage);
  uint64_t* empty = full + TS;
  uint64_t* done = empty + TS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int kt0 = blockIdx.z * kt_per;
  const int nk = max(0, min(ktiles, kt0 + kt_per) - kt0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < TS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)(Md::acc * TN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // producer: TMA ring
    int issued[TS] = {};
    for (int i = 0; i < nk; ++i) {
      const int s = i % TS;
      const uint32_t ph = (uint32_t)(i / TS) & 1u;
      if (i >= TS && !mbar_wait(&empty[s], ph ^ 1u, kWaitNs)) {
        atomicOr(status, 1u);
        break;
      }
      unsigned char* stg = base + (size_t)s * kStage;
      mbar_expect_tx(&full[s], kStage);
      const int x = (kt0 + i) * TK;
      if constexpr (BF16) {
        tma_load_2d(stg, &mAh, &full[s], x, m0);
        tma_load_2d(stg + kTileA, &mBh, &full[s], x, n0);
      } else {
        tma_load_2d(stg, &mAh, &full[s], x, m0);
        tma_load_2d(stg + kTileA, &mAl, &full[s], x, m0);
        tma_load_2d(stg + 2 * kTileA, &mBh, &full[s], x, n0);
        tma_load_2d(stg + 2 * kTileA + kTileB, &mBl, &full[s], x, n0);
      }
      issued[s] += 1;
    }
    // no copy of this CTA may still be landing when it exits
    for (int s = 0; s < TS; ++s)
      if (issued[s] && !mbar_wait(&full[s], (uint32_t)(issued[s] - 1) & 1u, kWaitNs))
        atomicOr(status, 4u);
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    for (int i = 0; i < nk; ++i) {
      const int s = i % TS;
      const uint32_t ph = (uint32_t)(i / TS) & 1u;
      if (!mbar_wait(&full[s], ph, kWaitNs)) {
        atomicOr(status, 2u);
        break;
      }
      tc_fence_after();
      const uint32_t ah = smem_u32(base + (size_t)s * kStage);
      const uint32_t d = tmem + (uint32_t)(i % Md::acc * TN);
      const bool more = i >= Md::acc;
      if constexpr (BF16) {
        const uint32_t bh = ah + kTileA;
#pragma unroll
        for (int kk = 0; kk < TK / Md::KMMA; ++kk) {
          const uint32_t off = kk * 32;  // 16 BF16 values
          umma_bf16(d, sdesc_sw128(ah + off), sdesc_sw128(bh + off), (more || kk > 0) ? 1u : 0u);
        }
      } else {
        const uint32_t al = ah + kTileA, bh = ah + 2 * kTileA, bl = bh + kTileB;
#pragma unroll
        for (int kk = 0; kk < TK / Md::KMMA; ++kk) {
          const uint32_t off = kk * 32;  // 8 TF32 values
          const uint64_t dah = sdesc_sw128(ah + off), dal = sdesc_sw128(al + off);
          const uint64_t dbh = sdesc_sw128(bh + off), dbl = sdesc_sw128(bl + off);
          umma_tf32(d, dah, dbh, (more || kk > 0) ? 1u : 0u);
          umma_tf32(d, dah, dbl, 1u);
          umma_tf32(d, dal, dbh, 1u);
        }
      }
      umma_commit(&empty[s]);
    }
    umma_commit(done);  // arrives once every MMA issued above has completed
  }
  __syncwarp();
  // epilogue: the done wait outlasts the producer's and the issuer's bounds
  const bool ok = mbar_wait(done, 0u, 4 * kWaitNs);
  __syncwarp();
  tc_fence_after();
  // The accumulators go to shared memory (no copy or MMA uses the stages any more), and
  // each CTA of the cluster stores a share of the rows.
  float* sums = reinterpret_cast<float*>(base);
  if (!ok && threadIdx.x == 0) atomicOr(status, 8u);
  for (int c = 0; c < TN; c += 16) {
    float v[16] = {};
    if (ok && nk > 0) {
      const uint32_t t = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c;
      tmem_ld16(t, v);
      for (int q = 1; q < min(nk, Md::acc); ++q) {
        float w[16];
        tmem_ld16(t + (uint32_t)(q * TN), w);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += w[j];
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) sums[(warp * 32 + lane) * kTcRow + c + j] = v[j];
  }
  tc_fence_before();
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)(Md::acc * TN))
                 : "memory");
  }
  const int nz = (int)cluster.num_blocks(), z = (int)cluster.block_rank();
  const int mv = min(TM, M - m0), per = (mv + nz - 1) / nz;
  const int r0 = z * per, r1 = min(mv, r0 + per), nc = min(TN, N - n0);
  const uint32_t at = smem_u32(sums);
  const bool add = !part && (alpha != 1.0 || beta != 0.0);
  const size_t ldo = part ? N : ldc;
  OutT* out = (part ? part + (size_t)(blockIdx.z / nz) * M * N : C) + (size_t)m0 * ldo + n0;
  switch (nz) {  // a power of two (host)
    case 1: tc_store<1, OutT>(at, r0, r1, nc, add, alpha, beta, out, ldo); break;
    case 2: tc_store<2, OutT>(at, r0, r1, nc, add, alpha, beta, out, ldo); break;
    case 4: tc_store<4, OutT>(at, r0, r1, nc, add, alpha, beta, out, ldo); break;
    default: tc_store<kTcCluster, OutT>(at, r0, r1, nc, add, alpha, beta, out, ldo); break;
  }
  cluster.sync();  // no CTA leaves while another reads its sums
}

__device__ __forceinline__ float tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// hi / lo FP32 parts of op(X) as a rows x kp K-contiguous array: element
// (r, k) is X[r * ldx + k] (trans = 0) or X[k * ldx + r] (trans = 1), zero for
// k >= K.  32 x 32 tiles through shared memory so both sides stay coalesced;
// blockIdx.z picks the operand.
struct TcOperand {
  const double* X;
  int ldx, rows, trans;
  void* hi;
  float* lo;
};
__global__ void k_split_tf32(TcOperand A, TcOperand B, int K, int kp) {
  const TcOperand& o = blockIdx.z ? B : A;
  const double* __restrict__ X = o.X;
  const int ldx = o.ldx, rows = o.rows, trans = o.trans;
  float *hi = reinterpret_cast<float*>(o.hi), *lo = o.lo;
  __shared__ double tile[32][33];
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  if (r0 >= rows) return;  // uniform over the block
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int j = ty; j < 32; j += 8) {
    double v = 0.0;
    if (trans) {  // read along r: tile[k][r]
      const int k = k0 + j, r = r0 + tx;
      if (k < K && r < rows) v = X[(size_t)k * ldx + r];
      tile[j][tx] = v;
    } else {  // read along k: tile[r][k]
      const int r = r0 + j, k = k0 + tx;
      if (k < K && r < rows) v = X[(size_t)r * ldx + k];
      tile[j][tx] = v;
    }
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j, k = k0 + tx;
    if (r < rows && k < kp) {
      const double v = trans ? tile[tx][j] : tile[j][tx];
      const float h = tf32_rna((float)v);
      hi[(size_t)r * kp + k] = h;
      lo[(size_t)r * kp + k] = (float)(v - (double)h);
    }
  }
}

// op(X) rounded to BF16 as a rows x kp K-contiguous array (same tiling and
// element rule as k_split_tf32).
__global__ void k_split_bf16(TcOperand A, TcOperand B, int K, int kp) {
  const TcOperand& o = blockIdx.z ? B : A;
  const double* __restrict__ X = o.X;
  const int ldx = o.ldx, rows = o.rows, trans = o.trans;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(o.hi);
  __shared__ double tile[32][33];
  const int r0 = blockIdx.y * 32, k0 = blockIdx.x * 32;
  if (r0 >= rows) return;  // uniform over the block
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int j = ty; j < 32; j += 8) {
    double v = 0.0;
    if (trans) {
      const int k = k0 + j, r = r0 + tx;
      if (k < K && r < rows) v = X[(size_t)k * ldx + r];
    } else {
      const int r = r0 + j, k = k0 + tx;
      if (k < K && r < rows) v = X[(size_t)r * ldx + k];
    }
    tile[j][tx] = v;
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j, k = k0 + tx;
    if (r < rows && k < kp)
      out[(size_t)r * kp + k] = __float2bfloat16_rn((float)(trans ? tile[tx][j] : tile[j][tx]));
  }
}

template <typename OutT>
__global__ void k_tc_reduce(int M, int N, int nz, const OutT* __restrict__ part, double alpha,
                            double beta, OutT* __restrict__ C, int ldc) {
  const size_t mn = (size_t)M * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < mn;
       e += (size_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int z = 0; z < nz; ++z) acc += (double)part[(size_t)z * mn + e];
    OutT* p = C + (e / N) * ldc + (e % N);
    *p = beta == 0.0 ? (OutT)(alpha * acc) : (OutT)fma(alpha, acc, beta * (double)*p);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
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

// 2-D map over a rows x kp K-contiguous plane (FP32 or BF16), box = one
// 128-byte slab row of box_rows rows, 128-byte swizzle.
int make_map(CUtensorMap* map, const void* base, bool bf16, int rows, int kp, int box_rows) {
  auto enc = encode_fn();
  if (!enc) {
    set_error("tensor-core GEMM: cuTensorMapEncodeTiled not available");
    return SM_ERR_CUDA;
  }
  const size_t es = bf16 ? 2 : 4;
  const cuuint64_t dims[2] = {(cuuint64_t)kp, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)kp * es};
  const cuuint32_t box[2] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                         2, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("tensor-core GEMM: tensor map encoding failed");
    return SM_ERR_CUDA;
  }
  return SM_OK;
}

}  // namespace

bool gemm_tc_eligible(int M, int N, int K) {
  // below a few tiles of work the SIMT FP32 kernel is as fast and has no
  // split step
  return (double)M * N * K >= 4.0 * 1024 * 1024 && M >= 64 && N >= 64 && K >= 32 &&
         encode_fn() != nullptr;
}

int tc_kslab(bool bf16) { return bf16 ? TcMode<true>::TK : TcMode<false>::TK; }

namespace {
// the planes of one operand, or of two in one launch
int split_planes(cudaStream_t st, const TcOperand& a, const TcOperand* b, int K, int kp, bool bf16) {
  const int rows = std::max(a.rows, b ? b->rows : 0);
  const dim3 blk(32, 8), grd(kp / 32, (rows + 31) / 32, b ? 2 : 1);
  if (bf16) k_split_bf16<<<grd, blk, 0, st>>>(a, b ? *b : a, K, kp);
  else k_split_tf32<<<grd, blk, 0, st>>>(a, b ? *b : a, K, kp);
  note_launch();
  SM_CUDA_CHECK(cudaGetLastError());
  return SM_OK;
}

template <typename... P, typename... Q>
int cluster_launch(void (*fn)(P...), dim3 grid, int block, int nz, size_t smem, cudaStream_t st,
                   Q... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 1;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = nz;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  SM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, fn, args...));
  return SM_OK;
}
}  // namespace

int tc_planes(Ctx&, cudaStream_t st, const double* X, int ldx, int rows, int K, int kp, int trans,
              bool bf16, void* hi, float* lo) {
  return split_planes(st, TcOperand{X, ldx, rows, trans, hi, lo}, nullptr, K, kp, bf16);
}

template <typename OutT>
int gemm_tc_planes(Ctx& ctx, cudaStream_t st, int M, int N, int kp, bool bf16, const void* ah,
                   const float* al, const void* bh, const float* bl, double alpha, double beta,
                   OutT* C, int ldc) {
  const int TK = tc_kslab(bf16);
  const int ktiles = kp / TK;
  unsigned int* status;
  SM_CHECK(tc_status(ctx, &status));
  CUtensorMap mAh, mAl, mBh, mBl;
  SM_CHECK(make_map(&mAh, ah, bf16, M, kp, TM));
  SM_CHECK(make_map(&mBh, bh, bf16, N, kp, TN));
  if (bf16) {
    mAl = mAh;
    mBl = mBh;
  } else {
    SM_CHECK(make_map(&mAl, al, false, M, kp, TM));
    SM_CHECK(make_map(&mBl, bl, false, N, kp, TN));
  }
  const int tiles = ((M + TM - 1) / TM) * ((N + TN - 1) / TN);
  // K over the CTAs of a cluster while the output has fewer tiles than SMs.  The tensor
  // cores truncate as they accumulate, an error that grows with the slabs an accumulator
  // takes: two slabs to an accumulator, and beyond that several clusters to a tile,
  // whose sum is another launch.
  const int sms = std::max(1, ctx.num_sms);
  const auto kernel = bf16 ? k_gemm_tc<true, OutT> : k_gemm_tc<false, OutT>;
  const size_t smem = bf16 ? TcMode<true>::smem : TcMode<false>::smem;
  SM_CHECK(raise_smem_limit(kernel, smem));
  int nmax = kTcCluster;  // the largest cluster that finds room
  while (nmax > 1 && !ctx.places(reinterpret_cast<const void*>(kernel), nmax, kTCThreads, smem)) nmax /= 2;
  int nz = 1, nzo = 1, kt_per;
  if (bf16) {  // ranges of two slabs and more, an accumulator each
    const int want = std::max(1, std::min(sms / tiles, ktiles / 2));
    kt_per = (ktiles + want - 1) / want;
    const int ranges = (ktiles + kt_per - 1) / kt_per;
    while (nz < nmax && nz < ranges) nz *= 2;
    nzo = (ranges + nz - 1) / nz;
  } else {
    while (nz < nmax && 2 * nz <= std::min(sms / tiles, ktiles)) nz *= 2;
    // Two CTAs share a tile from more slabs on than one's accumulators take two of: a call
    // of 1200 x 69 x 85 takes 40 us in one CTA a tile and 50 in two, 1024 x 1024 x 256 46
    // and 52 (x 512 52 and 56, x 1024 75 and 68).
    if (nz == 2 && ktiles <= 2 * TcMode<false>::acc) nz = 1;
    kt_per = (ktiles + nz - 1) / nz;
    constexpr int most = 2 * TcMode<false>::acc;
    if (nz == nmax)
      nzo = std::max(1, std::min(sms / (tiles * nz), (kt_per + most - 1) / most));
    if (nzo > 1) kt_per = (ktiles + nz * nzo - 1) / (nz * nzo);
  }
  OutT* part = nullptr;
  if (nzo > 1)
    SM_CHECK(ctx.scratch(sizeof(OutT) == 8 ? "tc.part" : "tc.part32", (size_t)nzo * M * N, &part));
  const dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM, nz * nzo);
  SM_CHECK(cluster_launch(kernel, grid, kTCThreads, nz, smem, st, mAh, mAl, mBh, mBl, M, N, ktiles,
                          kt_per, alpha, beta, C, ldc, part, status));
  note_launch();
  if (nzo > 1) {
    const size_t mn = (size_t)M * N;
    k_tc_reduce<OutT><<<(int)std::min<size_t>((mn + 255) / 256, 4096), 256, 0, st>>>(
        M, N, nzo, part, alpha, beta, C, ldc);
    note_launch();
    SM_CUDA_CHECK(cudaGetLastError());
  }
  return SM_OK;
}

template int gemm_tc_planes<double>(Ctx&, cudaStream_t, int, int, int, bool, const void*,
                                    const float*, const void*, const float*, double, double,
                                    double*, int);
template int gemm_tc_planes<float>(Ctx&, cudaStream_t, int, int, int, bool, const void*,
                                   const float*, const void*, const float*, double, double, float*,
                                   int);

int gemm_tc(Ctx& ctx, cudaStream_t st, int opA, int opB, int M, int N, int K, double alpha,
            const double* A, int lda, const double* B, int ldb, double beta, double* C, int ldc,
            bool bf16) {
  const int TK = tc_kslab(bf16);
  const int kp = (K + TK - 1) / TK * TK;
  // op(A)[m][k]: A[m][k] (N) or A[k][m] (T, C: real); op(B)^T[n][k]: B[k][n]
  // (N) or B[n][k] (T, C)
  const int ta = opA == SM_OP_N ? 0 : 1, tb = opB == SM_OP_N ? 1 : 0;
  void *ah, *bh;
  float *al = nullptr, *bl = nullptr;
  const size_t es = bf16 ? 2 : 4;
  SM_CHECK(ctx.scratch(bf16 ? "tc.Abf" : "tc.Ah", es * (size_t)M * kp, &ah));
  SM_CHECK(ctx.scratch(bf16 ? "tc.Bbf" : "tc.Bh", es * (size_t)N * kp, &bh));
  if (!bf16) {
    SM_CHECK(ctx.scratch("tc.Al", (size_t)M * kp, &al));
    SM_CHECK(ctx.scratch("tc.Bl", (size_t)N * kp, &bl));
  }
  const TcOperand oa{A, lda, M, ta, ah, al}, ob{B, ldb, N, tb, bh, bl};
  SM_CHECK(split_planes(st, oa, &ob, K, kp, bf16));
  return gemm_tc_planes<double>(ctx, st, M, N, kp, bf16, ah, al, bh, bl, alpha, beta, C, ldc);
}

int tc_status(Ctx& ctx, unsigned int** out) {
  auto it = ctx.bufs.find("tc.status");
  const bool fresh = it == ctx.bufs.end();
  SM_CHECK(ctx.scratch("tc.status", sizeof(unsigned int), reinterpret_cast<void**>(out)));
  if (fresh) SM_CUDA_CHECK(cudaMemset(*out, 0, sizeof(unsigned int)));
  return SM_OK;
}

int tc_status_check(Ctx& ctx, cudaStream_t st) {
  if (ctx.bufs.find("tc.status") == ctx.bufs.end()) return SM_OK;
  unsigned int* status;
  SM_CHECK(tc_status(ctx, &status));
  unsigned int* h = reinterpret_cast<unsigned int*>(ctx.pinned) + 1000;
  SM_CUDA_CHECK(cudaMemcpyAsync(h, status, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
  SM_CUDA_CHECK(cudaStreamSynchronize(st));
  if (*h) {
    SM_CUDA_CHECK(cudaMemsetAsync(status, 0, sizeof(unsigned int), st));
    set_error("tensor-core GEMM: a pipeline wait timed out (status " + std::to_string(*h) + ")");
    return SM_ERR_CUDA;
  }
  return SM_OK;
}

}  // namespace sm
