// FP32 stage of the splits, second half: block-cyclic one-sided Jacobi on the rows of
// R in one thread-block cluster.
//
// The rows are cut into 2 C blocks of r <= 16 rows (C CTAs); CTA c holds the blocks
// "top" c and "bottom" 2C - 1 - c in shared memory.  A sweep rotates the pairs inside
// each block once, then makes 2C - 1 block rounds: r local rounds in which warp w
// keeps top row w in registers and the bottom rows come by, after which the tops move
// one CTA up and the bottoms one CTA down (the round-robin of 2C players).
//
// What bounds it is latency: a local round is a chain of a shared-memory load, one dot
// product with its warp sum, the angle and the rotation (~500 clocks), and there are
// r (2C - 1) of them per sweep however the rows are cut.  So
//   * the cluster is the smallest whose blocks have at most 8 rows (16 in the largest):
//     fewer block rounds, until the warps of a scheduler hinder each other (a local
//     round takes 630 clocks with 10 warps, 950 with 16);
//   * only the overlap is summed in a local round; the rows' norms are taken afresh
//     once per block round and follow the rotations within it;
//   * four warps share a scheduler, so instructions count as much as latency: FP32
//     arithmetic is issued in pairs (f32x2), the angle takes two reciprocal roots of
//     the SFU, and convergence is a flag (did a rotation start
//     above the stopping cosine), not a maximum;
//   * after the last local round each warp copies its two rows into the next CTAs'
//     buffers (bulk copies), and a CTA waits on its own mbarrier for the bytes of
//     its new blocks: no cluster barrier.  Two buffers per block are enough: a CTA
//     has sent round g's rows only after all its warps are done with the buffers of
//     round g - 1, and its neighbours send into those only after they have received
//     rows of it.  The rows leave from two more buffers per block, free again two rounds
//     later: by then the CTA has received rows that its neighbours sent after they had
//     its own.  Where shared memory holds four buffers a block only, they leave from the
//     round's own.  These are written over a round later, by a neighbour that need not
//     have received them (a top goes up while its place is filled from below), and a
//     copy is known to have read its source only where it arrives: whoever has received
//     a round's rows tells the CTAs that write over their sources (an mbarrier each,
//     sync_rules.h).  Reports cost up to a tenth: a sweep on 153 rows of 256 takes 63 us
//     with the buffers apart and 68 with reports, on 256 rows 100 and 107, on 337 rows of
//     512 210 and 217.  (They are made by a warp without a row where there is one, 4 to
//     10 % less than by a warp of the pairs: their arrivals release to the cluster.)
// The cluster meets once per sweep, to agree on that flag.  A sweep takes 21 us on 64
// rows of 64, 63 us on 153 rows of 256 and 210 us on 337 rows of 512 (with 16 CTAs
// always, three sums per pair, copies through mailboxes and a cluster barrier per
// block round: 56, 93 and 268 us).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "svd_cluster.cuh"
#include "sync_rules.h"

namespace cg = cooperative_groups;

namespace sm {

namespace {

// A sweep whose rotations all start below cosine 1e-2 ends the iteration:
// convergence is quadratic, so the rows leave it orthogonal to ~1e-4 / gap, which the
// FP64 steps after it take to FP64 level for less than another sweep costs.
constexpr float kStopC2 = 1e-4f;
// R has norm 1: rows of squared norm below kTinyRow2 are left alone (no rank rule sees
// them), and a pair is rotated only if its |g|^2 relative to the larger squared norm
// is above kTinyG2 (clear of the SFU's subnormal flush)
constexpr float kTinyRow2 = 1e-30f;
constexpr float kTinyG2 = 1e-36f;

struct JacShared {
  uint64_t bar[2];             // this CTA's new blocks, by the round's parity
  uint64_t clear[2];           // a round's copies out of the buffers this CTA writes next
  float nB[2][16];             // squared norms of the bottom rows, by the round's parity
  int verdict[2][kCWMax];      // every CTA's rotations of the sweep, by its parity: 1 some
                               //   above the stopping cosine, 2 a wait ran out
};

__device__ __forceinline__ void pair_barrier(int warps) {  // the warps that hold a row
  asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
}

// E row elements per lane (a row is padded to 32 E)
template <typename T, int E>
__global__ void __launch_bounds__(kCNT, 1)
    k_jacobi_cluster(const typename F32<T>::type* __restrict__ Rg, int ldk, int kmax, int l,
                     float tol2, int max_sweeps, uint32_t smem, T* __restrict__ out_rows,
                     double* __restrict__ out_nrm, int kcap, JacobiCtl* ctl,
                     double* __restrict__ info) {
  using F = typename F32<T>::type;
  constexpr bool kCplx = sizeof(F) == 8;
  constexpr int LP = 32 * E;                         // elements of a padded row
  constexpr int NU = E * (int)sizeof(F) / 8;         // 64-bit pairs of a row per lane
  constexpr uint32_t kRowBytes = LP * sizeof(F);
  extern __shared__ __align__(16) unsigned char jac_raw[];
  __shared__ JacShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), nc = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long t_start = global_ns();
  const int keff = ctl->nact;
  if (ctl->status != 0) return;  // the QR gave up (every CTA reads the same word)
  const int r = max(1, (keff + 2 * nc - 1) / (2 * nc));
  const uint32_t blk = (uint32_t)r * kRowBytes;
  // where a round's rows are copied from, behind its buffers: others, or themselves
  const bool apart = 8 * blk <= smem;
  // block buffers [top / bottom][parity]
  auto buf = [&](int half, int par) -> unsigned char* {
    return jac_raw + (size_t)(half * 2 + par) * blk;
  };
  if (tid == 0) {
    cl_mbar_init(&sh.bar[0], 1);
    cl_mbar_init(&sh.bar[1], 1);
    cl_mbar_init(&sh.clear[0], max(1, jac_reports(rank, nc)));
    cl_mbar_init(&sh.clear[1], max(1, jac_reports(rank, nc)));
    cl_mbar_fence();
  }
  // ---- the rows of R (column-major in L2; zero rows past keff) ------------------
  for (int half = 0; half < 2; ++half) {
    const int row0 = (half ? 2 * nc - 1 - rank : rank) * r;
    F* dst = reinterpret_cast<F*>(buf(half, 0));
    for (int f = tid; f < r * LP; f += kCNT) {
      const int x = f / r, ri = f % r;  // consecutive threads: consecutive rows of a column
      F v = F32<T>::zero();
      if (x < l && row0 + ri < keff) v = Rg[(size_t)x * ldk + row0 + ri];
      dst[(size_t)ri * LP + x] = v;
    }
  }
  cluster.sync();  // barriers initialised, before any row is sent
  const uint32_t base = cl_smem(jac_raw);
  auto adr = [&](int half, int par) { return base + (uint32_t)(half * 2 + par) * blk; };
  // a row as 16-byte vectors: lane holds bytes 16 lane .. of every 512
  auto load_row = [&](uint32_t row, f2_t* x) {
#pragma unroll
    for (int e = 0; e < NU / 2; ++e) cl_lds16(row + (uint32_t)(lane + 32 * e) * 16u, x[2 * e], x[2 * e + 1]);
  };
  auto store_row = [&](uint32_t row, const f2_t* x) {
#pragma unroll
    for (int e = 0; e < NU / 2; ++e) cl_sts16(row + (uint32_t)(lane + 32 * e) * 16u, x[2 * e], x[2 * e + 1]);
  };
  auto norm2_of = [&](const f2_t* u) {
    f2_t s0 = f2_mul(u[0], u[0]), s1 = f2_mul(u[1], u[1]);
#pragma unroll
    for (int e = 2; e < NU; e += 2) {
      s0 = f2_fma(u[e], u[e], s0);
      s1 = f2_fma(u[e + 1], u[e + 1], s1);
    }
    return warp_sum(f2_hsum(f2_add(s0, s1)));
  };
  // conj(u) v
  auto dot_of = [&](const f2_t* u, const f2_t* v, float& gr, float& gi) {
    f2_t s0 = f2_mul(u[0], v[0]), s1 = f2_mul(u[1], v[1]);
#pragma unroll
    for (int e = 2; e < NU; e += 2) {
      s0 = f2_fma(u[e], v[e], s0);
      s1 = f2_fma(u[e + 1], v[e + 1], s1);
    }
    gr = f2_hsum(f2_add(s0, s1));
    gi = 0.f;
    if constexpr (kCplx) {  // im(conj(p) q) = p.x q.y - p.y q.x
      f2_t t0 = f2_mul(u[0], f2_mul_mi(v[0])), t1 = f2_mul(u[1], f2_mul_mi(v[1]));
#pragma unroll
      for (int e = 2; e < NU; e += 2) {
        t0 = f2_fma(u[e], f2_mul_mi(v[e]), t0);
        t1 = f2_fma(u[e + 1], f2_mul_mi(v[e + 1]), t1);
      }
      gi = f2_hsum(f2_add(t0, t1));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      gr += __shfl_xor_sync(0xffffffffu, gr, o);
      if constexpr (kCplx) gi += __shfl_xor_sync(0xffffffffu, gi, o);
    }
  };
  bool wide = false;  // a rotation of this warp in the sweep started above the stopping cosine
  // Rotates the register rows u (squared norm a) and v (b) so that conj(u) v becomes
  // zero; the norms follow.  False if the pair is orthogonal already.
  auto rotate = [&](f2_t* u, f2_t* v, float& a, float& b) -> bool {
    float gr, gi;
    dot_of(u, v, gr, gi);
    // The angle depends on a : b : g only: everything is scaled by the power of two
    // that brings the larger squared norm to [1, 2), so that rows far below |W| (whose
    // a b and g^2 leave the FP32 range) are rotated like the others.
    const float sc = __int_as_float(0x7f000000 - (__float_as_int(fmaxf(a, b)) & 0x7f800000));
    const float xr = gr * sc, xi = gi * sc, ab = (a * sc) * (b * sc);
    const float g2 = kCplx ? fmaf(xr, xr, xi * xi) : xr * xr;
    if (!(g2 > fmaxf(kTinyG2, tol2 * ab) && fminf(a, b) >= kTinyRow2)) return false;
    wide = wide || g2 >= kStopC2 * ab;
    // with R = sqrt(d^2 + 4|g|^2), d = b - a: cos^2 = (1 + |d| / R) / 2 and
    // sin = sign(d) |g| / (R cos), times g's phase: two reciprocal roots
    const float d = (b - a) * sc;
    const float ir = f_rsqrt(fmaf(d, d, 4.0f * g2));
    const float cc = fmaf(0.5f * fabsf(d), ir, 0.5f);
    const float rc = f_rsqrt(cc), c = cc * rc, sr = copysignf(ir * rc, d);
    const float ar = xr * sr, ai = xi * sr;
    const float dn = rc * (kCplx ? fmaf(ar, gr, ai * gi) : ar * gr);  // tan |g|
    a = fmaxf(a - dn, 0.f);
    b = fmaxf(b + dn, 0.f);
    const f2_t c2 = f2_pack(c, c), r2 = f2_pack(ar, ar), m2 = f2_pack(-ar, -ar);
    if constexpr (!kCplx) {
#pragma unroll
      for (int e = 0; e < NU; ++e) {
        const f2_t p = u[e], w = v[e];
        u[e] = f2_fma(m2, w, f2_mul(c2, p));  // c p - s q
        v[e] = f2_fma(r2, p, f2_mul(c2, w));  // s p + c q
      }
    } else {  // p' = c p - conj(s e) q ; q' = (s e) p + c q
      const f2_t mi = f2_pack(-ai, -ai);
#pragma unroll
      for (int e = 0; e < NU; ++e) {
        const f2_t p = u[e], w = v[e];
        u[e] = f2_fma(mi, f2_mul_mi(w), f2_fma(m2, w, f2_mul(c2, p)));
        v[e] = f2_fma(mi, f2_mul_mi(p), f2_fma(r2, p, f2_mul(c2, w)));
      }
    }
    return true;
  };
  // where the blocks go
  const JacBlock tdst = jac_dest(rank, 0, nc), bdst = jac_dest(rank, 1, nc);
  const bool top_stays = tdst.cta == rank;
  const uint32_t incoming = (top_stays ? 1u : 2u) * blk;
  bool timeout = false;
  // the rows of round gr are here
  auto tell = [&](unsigned int gr) {
    const int report = lane < 2 ? jac_report(rank, lane, nc) : -1;
    if (report >= 0 && !timeout) cl_mbar_arrive(cl_map(cl_smem(&sh.clear[gr & 1]), report));
  };
  unsigned int g = 0;  // block rounds so far; the active buffers have parity g & 1
  // A sweep's block rounds for the warps that hold rows, in one of the two ways to send
  // them (compiled apart: the one's registers and branches would slow the other).
  auto block_rounds = [&](auto way) {
    constexpr bool kApart = decltype(way)::value;
    const uint32_t out = kApart ? 4 * blk : 0;
    const bool reported = !kApart && jac_reports(rank, nc) > 0;
    for (int br = 0; br < 2 * nc - 1; ++br, ++g) {
      const int ap = g & 1, np = ap ^ 1;
      if (tid == 0) cl_mbar_expect(&sh.bar[ap], incoming);
      const uint32_t B = adr(1, ap), nB = cl_smem(sh.nB[ap]);
      f2_t tr[NU], v[NU];
      load_row(adr(0, ap) + (uint32_t)warp * kRowBytes, tr);
      load_row(B + (uint32_t)warp * kRowBytes, v);
      float a = norm2_of(tr);
      {
        const float b = norm2_of(v);
        if (lane == 0) cl_sts(nB + 4u * warp, b);
      }
      pair_barrier(r);
      uint32_t brow = B + (uint32_t)warp * kRowBytes, nb = nB + 4u * warp;
      const uint32_t bend = B + blk;
#pragma unroll 1
      for (int t = r; t > 0; --t) {
        load_row(brow, v);
        float b = cl_lds(nb);
        const bool rot = rotate(tr, v, a, b);
        if (t == 1) break;
        if (rot) {
          store_row(brow, v);
          if (lane == 0) cl_sts(nb, b);
        }
        pair_barrier(r);
        brow += kRowBytes;
        nb += 4;
        if (brow == bend) {
          brow = B;
          nb = nB;
        }
      }
      // Both rows to where they meet next, one bulk copy each.  CTA 0's top and the
      // last CTA's top (its own bottom next) stay in the CTA: plain stores of the warp
      // that reads them first.
      const uint32_t trow = adr(0, ap) + out + (uint32_t)warp * kRowBytes;
      store_row(brow + out, v);
      if (!top_stays) store_row(trow, tr);
      cl_bulk_fence();
      // without buffers apart those written now were the sources of the round before
      if (reported && g > 0 && !timeout && !cl_mbar_wait(&sh.clear[np], ((g - 1) >> 1) & 1))
        timeout = true;
      __syncwarp();
      if (top_stays) store_row(adr(tdst.half, np) + (uint32_t)warp * kRowBytes, tr);
      if (lane == 0 && !timeout) {
        const uint32_t bar = cl_smem(&sh.bar[ap]);
        if (!top_stays)
          cl_bulk(cl_map(adr(tdst.half, np) + (uint32_t)warp * kRowBytes, tdst.cta), trow, kRowBytes,
                  cl_map(bar, tdst.cta));
        cl_bulk(cl_map(adr(bdst.half, np) + (brow - B), bdst.cta), brow + out, kRowBytes,
                cl_map(bar, bdst.cta));
      }
      if (!timeout && !cl_mbar_wait(&sh.bar[ap], (g >> 1) & 1)) timeout = true;
      if (!kApart && r == kCNW && warp == 0) tell(g);
    }
  };
  int status = DEV_NOT_CONVERGED, sweeps = max_sweeps;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    wide = false;
    // pairs inside each block (circle method over r positions, padded to even)
    {
      const int rp2 = r + (r & 1), half_n = rp2 / 2;
      const uint32_t blk0 = adr(warp / 8, g & 1);
      const int w8 = warp % 8;
      int p = w8 == 0 ? rp2 - 1 : w8, q = w8 == 0 ? 0 : rp2 - 1 - w8;  // round t adds t mod (rp2 - 1)
#pragma unroll 1
      for (int t = 0; t < rp2 - 1; ++t) {
        if (w8 < half_n && p < r && q < r) {
          const uint32_t pa = blk0 + (uint32_t)p * kRowBytes, qa = blk0 + (uint32_t)q * kRowBytes;
          f2_t u[NU], v[NU];
          load_row(pa, u);
          load_row(qa, v);
          float a = norm2_of(u), b = norm2_of(v);
          if (rotate(u, v, a, b)) {
            store_row(pa, u);
            store_row(qa, v);
          }
        }
        if (w8 != 0) p = p + 1 == rp2 - 1 ? 0 : p + 1;
        q = q + 1 == rp2 - 1 ? 0 : q + 1;
        __syncthreads();
      }
    }
    if (warp < r) {
      if (apart) block_rounds(std::true_type());
      else block_rounds(std::false_type());
    } else if (!apart && warp == r && (jac_report(rank, 0, nc) >= 0 || jac_report(rank, 1, nc) >= 0)) {
      for (int br = 0; br < 2 * nc - 1; ++br, ++g) {
        if (lane < 2 && !timeout && !cl_mbar_wait(&sh.bar[g & 1], (g >> 1) & 1)) timeout = true;
        tell(g);
      }
      __syncwarp();
    } else {
      g += 2 * nc - 1;
    }
    // the sweep's verdict, over the cluster
    const int mine = __syncthreads_or(wide ? 1 : 0) ? 1 : 0;
    const int ran_out = __syncthreads_or(timeout ? 1 : 0) ? 2 : 0;
    if (tid < nc) cluster.map_shared_rank(&sh, tid)->verdict[sweep & 1][rank] = mine | ran_out;
    cluster.sync();
    int all = 0;
    for (int c = 0; c < nc; ++c) all |= sh.verdict[sweep & 1][c];
    if (all & 2) {  // the whole cluster stops
      status = DEV_BARRIER_TIMEOUT;
      break;
    }
    if (!all) {
      status = 0;
      sweeps = sweep + 1;
      break;
    }
  }
  // ---- rows back to global memory (FP64, rescaled by |W|) -----------------------
  const double nrm = sqrt(info[0]);
  for (int j = warp; j < 2 * r; j += kCNW) {
    const int half = j >= r, row = rank * 2 * r + j;
    if (row >= kcap) continue;
    const F* src = reinterpret_cast<const F*>(buf(half, g & 1)) + (size_t)(j - half * r) * LP;
    double acc = 0.0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int c = lane + 32 * e;
      if (c < l) {
        const T x = F32<T>::to(src[c], nrm);
        out_rows[(size_t)row * l + c] = x;
        acc += S<T>::abs2(x);
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) out_nrm[row] = sqrt(acc);
  }
  for (int row = 2 * nc * r + rank * kCNW + warp; row < kcap; row += nc * kCNW) {
    for (int c = lane; c < l; c += 32) out_rows[(size_t)row * l + c] = S<T>::zero();
    if (lane == 0) out_nrm[row] = 0.0;
  }
  if (rank == 0 && tid == 0) {
    ctl->status = status;
    ctl->sweeps = sweeps;
    info[6] = 1e-6 * (double)(global_ns() - t_start);
  }
  cluster.sync();  // no CTA leaves while another may still store into its shared memory
}

// Elements per lane of a row (a multiple of 4: rows move as 16-byte vectors).
inline int e_bucket(int l) {
  const int need = (l + 31) / 32;
  for (int b : {4, 8, 12, 16, 24})
    if (need <= b) return b;
  return 0;
}

constexpr size_t kJacSmem = 225 * 1024;

// CTAs for kmax rows of length l: the fewest whose blocks have at most 8 rows, 16
// CTAs with up to 16 rows beyond that, if four block buffers fit shared memory (0: they
// do not); *smem: that of eight, or all there is
template <typename T>
int jac_ctas(int kmax, int l, size_t* smem) {
  for (int nc : {2, 4, 8, 16}) {
    const size_t r = (size_t)std::max(1, (kmax + 2 * nc - 1) / (2 * nc));
    const size_t block = r * 32 * e_bucket(l) * sizeof(typename F32<T>::type);
    *smem = std::min(8 * block, kJacSmem);
    if ((r <= 8 || (nc == 16 && r <= 16)) && 4 * block <= kJacSmem) return nc;
  }
  return 0;
}

// use(kernel) with the kernel for rows of length l; `none` beyond its sizes
template <typename T, typename Use, typename R>
R with_jacobi_kernel(int l, Use use, R none) {
  switch (e_bucket(l)) {
    case 4: return use(k_jacobi_cluster<T, 4>);
    case 8: return use(k_jacobi_cluster<T, 8>);
    case 12: return use(k_jacobi_cluster<T, 12>);
    case 16: return use(k_jacobi_cluster<T, 16>);
    case 24:
      if constexpr (sizeof(T) == sizeof(double)) return use(k_jacobi_cluster<T, 24>);
      return none;  // complex rows beyond 512 spill
    default: return none;
  }
}

}  // namespace

template <typename T>
bool jacobi_cluster_ok(Ctx& ctx, int kmax, int l) {
  if (kmax < 1) return false;
  return with_jacobi_kernel<T>(
      l,
      [&](auto fn) {
        size_t smem = 0;
        const int nc = jac_ctas<T>(kmax, l, &smem);
        return nc > 0 && cl_places(ctx, fn, nc, smem);
      },
      false);
}

template <typename T>
int jacobi_cluster(cudaStream_t st, const typename F32<T>::type* Rg, int ldk, int kmax, int l,
                   int max_sweeps, T* out_rows, double* out_nrm, int kcap, JacobiCtl* ctl,
                   double* info) {
  const float tol2 = (float)l * FLT_EPSILON * FLT_EPSILON;
  const int rc = with_jacobi_kernel<T>(
      l,
      [&](auto fn) {
        size_t smem = 0;
        const int nc = jac_ctas<T>(kmax, l, &smem);
        return cl_launch(fn, nc, smem, st, Rg, ldk, kmax, l, tol2, max_sweeps, (uint32_t)smem, out_rows,
                         out_nrm, kcap, ctl, info);
      },
      (int)SM_ERR_VALUE);
  if (rc == SM_ERR_VALUE) set_error("mixed split: row length beyond the cluster kernel's limit");
  return rc;
}

template int jacobi_cluster<double>(cudaStream_t, const float*, int, int, int, int, double*, double*,
                                    int, JacobiCtl*, double*);
template int jacobi_cluster<cplx>(cudaStream_t, const float2*, int, int, int, int, cplx*, double*,
                                  int, JacobiCtl*, double*);

// ---- the stage as one call ---------------------------------------------------------
// The sizes the stage takes (shared memory aside).
template <typename T>
bool split_cluster_size_ok(int kw, int l) {
  if (std::min(kw, l) > kMaxRows || kw > kMaxCol) return false;
  const int e = e_bucket(l);
  return e != 0 && (sizeof(T) == sizeof(double) || e <= 16);
}

template <typename T>
bool split_cluster_fits(Ctx& ctx, int kw, int l) {
  return split_cluster_size_ok<T>(kw, l) && qr_cluster_ok<T>(ctx, kw, l) &&
         jacobi_cluster_ok<T>(ctx, std::min(kw, l), l);
}

size_t split_cluster_rbuf_bytes(int kw, int l) {
  // R column-major, rows padded to whole vectors (the complex padding covers both)
  return (size_t)l * std::max(qr_row_pad<double>(kw) * sizeof(float), qr_row_pad<cplx>(kw) * sizeof(float2));
}

template <typename T>
int split_cluster_f32(cudaStream_t st, const T* A, int m, int n, bool want_u, double thr_rel,
                      double thr_abs, int max_sweeps, T* out_rows, double* out_nrm, int kcap,
                      JacobiCtl* ctl, double* info, int qr_cap, void* rbuf, bool pivot,
                      const int* cap_dev, bool plateau) {
  using F = typename F32<T>::type;
  // W = A^T (kw = n, l = m) when U is wanted, else W = A (kw = m, l = n)
  const int kw = want_u ? n : m, l = want_u ? m : n;
  F* Rg = reinterpret_cast<F*>(rbuf);
  SM_CHECK(qr_cluster<T>(st, A, n, want_u ? 1 : 0, kw, l, thr_rel, thr_abs, Rg, ctl, info, qr_cap,
                         cap_dev, pivot ? 1 : 0, plateau ? 1 : 0));
  const int kmax = qr_cap > 0 ? std::min(std::min(kw, l), qr_cap) : std::min(kw, l);
  return jacobi_cluster<T>(st, Rg, qr_row_pad<T>(kw), kmax, l, max_sweeps, out_rows, out_nrm, kcap,
                           ctl, info);
}

template bool split_cluster_size_ok<double>(int, int);
template bool split_cluster_size_ok<cplx>(int, int);
template bool split_cluster_fits<double>(Ctx&, int, int);
template bool split_cluster_fits<cplx>(Ctx&, int, int);
template int split_cluster_f32<double>(cudaStream_t, const double*, int, int, bool, double,
                                       double, int, double*, double*, int, JacobiCtl*, double*,
                                       int, void*, bool, const int*, bool);
template int split_cluster_f32<cplx>(cudaStream_t, const cplx*, int, int, bool, double, double,
                                     int, cplx*, double*, int, JacobiCtl*, double*, int, void*,
                                     bool, const int*, bool);

}  // namespace sm
