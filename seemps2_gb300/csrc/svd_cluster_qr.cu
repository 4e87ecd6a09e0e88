// FP32 stage of the splits, first half: rank-revealing Householder QR in one
// thread-block cluster, every column of W in the registers of one warp.
//
// A reflector is a chain (norm of the pivot column, broadcast, one dot product and
// one update per column), so what bounds the factorisation is the latency of that
// chain, not the chip's FP32 rate: kept in shared memory and blocked by 8 columns
// with a CTA-wide panel, a step of a 512 x 512 matrix took ~3 us (update, panel and
// pivoting a third each), and ~2.4 us even on 128 rows.  Here
//   * a warp owns NC columns, a lane 16-byte vectors of rows: dot products and
//     updates run in registers, and no column ever moves (pivoting only picks the
//     next owner; R is written in W's own column order);
//   * the owner of the next pivot column, as soon as it has applied a reflector,
//     forms its own and copies it into every CTA's ring of 8 (one bulk copy per CTA,
//     counted by an mbarrier there; 16-byte remote stores from the one warp took
//     ~30 clocks each, 1300 of a step's 2300 on 256 rows): a step waits for one
//     transfer, never for a barrier;
//   * the cluster meets once per 8 steps, to free the ring, to test the trailing
//     weight (once it is below the threshold, that of each of the 8 steps: a later
//     reflector leaves the weight below an earlier step unchanged) and to pick the 8 live columns of largest remaining weight
//     as the next pivots (block column pivoting).  Every CTA sends its 8 heaviest
//     to all and ranks the 128 candidates by counting, with no serial selection.
// 64 steps of 64 x 64 take 0.06 ms (blocked: 0.20), 153 of 256 x 256 0.20 (0.48), 337 of
// 512 x 512 0.67 (1.13).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "svd_cluster.cuh"

namespace cg = cooperative_groups;

namespace sm {

namespace {

constexpr int kRing = 8;  // steps per cluster barrier
// a column whose part below its pivot has norm <= kTinyCol (W has norm 1) gets no
// reflector: the part, weight <= 1e-30, is dropped, and tau would approach the FP32
// range; the QR also stops once the trailing weight is below kQrFloor
constexpr float kTinyCol = 1e-15f;
constexpr float kQrFloor = 1e-24f;
constexpr float kNoise = 1e-11f;  // trailing weight that FP32 noise does not exceed
constexpr float kFlat = 0.75f;    // its ratio over 8 pivots from which it counts as noise

struct QrShared {
  uint64_t full[kRing];
  float part[2][kCWMax][kRing];   // trailing-weight partials of all CTAs, by batch parity
  // heaviest columns of all CTAs: weight (float bits, negative: none) above ~column, so
  // that a larger key is a heavier column, or a smaller one of the same weight
  __align__(16) long long cand[2][kCWMax * kRing];
  __align__(16) long long mine[kRing];  // this CTA's 8 heaviest
  float wsum[kCNW][kRing];
  __align__(16) int cn[3 * kCNW];  // weight of this CTA's columns (float bits, negative: taken)
  int ord[kRing];                 // the batch's pivot columns
  double p64[kCWMax], red64[kCNW];
};

// elements of a 16-byte vector
__device__ __forceinline__ void vec_get(float4 t, float* v) {
  v[0] = t.x;
  v[1] = t.y;
  v[2] = t.z;
  v[3] = t.w;
}
__device__ __forceinline__ void vec_get(float4 t, float2* v) {
  v[0] = make_float2(t.x, t.y);
  v[1] = make_float2(t.z, t.w);
}
__device__ __forceinline__ float4 vec_put(const float* v) {
  return make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ float4 vec_put(const float2* v) {
  return make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
}
__device__ __forceinline__ float shfl_F(float v, int src) {
  return __shfl_sync(0xffffffffu, v, src);
}
__device__ __forceinline__ float2 shfl_F(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ float im_F(float) { return 0.f; }
__device__ __forceinline__ float im_F(float2 v) { return v.y; }
__device__ __forceinline__ float re_F(float v) { return v; }
__device__ __forceinline__ float re_F(float2 v) { return v.x; }
__device__ __forceinline__ void set_F(float& x, float re, float) { x = re; }
__device__ __forceinline__ void set_F(float2& x, float re, float im) { x = make_float2(re, im); }

// NV 16-byte vectors of rows per lane (row VW (lane + 32 e) + q), NC columns per warp
template <typename T, int NV, int NC>
__global__ void __launch_bounds__(kCNT, 1)
    k_qr_cluster(const T* __restrict__ A, int n_a, int trans, int kw, int l, double thr_rel,
                 double thr_abs, typename F32<T>::type* __restrict__ Rg, JacobiCtl* ctl_out,
                 double* __restrict__ info, int qr_cap, const int* __restrict__ cap_dev, int pivot,
                 int plateau) {
  using F = typename F32<T>::type;
  constexpr int VW = 16 / (int)sizeof(F);
  constexpr int VR = 32 * VW;        // rows of one vector index over the lanes
  constexpr int RP = VR * NV;        // padded rows
  constexpr bool kKeep = NV * 4 * (NC + 1) <= 64;  // registers for the reflector too
  constexpr int kSlot = 16 + NV * 512;  // tau, and a reflector
  extern __shared__ __align__(16) unsigned char ring_raw[];  // 8 slots, then their staging
  __shared__ QrShared sh;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), nc = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kmax = min(kw, l);
  if (cap_dev) qr_cap = cap_dev[0];  // a cap the rank predictor left on the device
  const int qsteps = qr_cap > 0 ? min(kmax, qr_cap) : kmax;
  auto col_of = [&](int s) { return rank * (kCNW * NC) + s * kCNW + warp; };
  auto row_of = [&](int e, int q) { return VW * (lane + 32 * e) + q; };
  const unsigned long long t_start = global_ns();
  if (tid == 0) {
    for (int i = 0; i < kRing; ++i) cl_mbar_init(&sh.full[i], 1);
    cl_mbar_fence();
  }
  auto Wat = [&](int i, int c) -> T {
    return trans ? A[(size_t)c * n_a + i] : A[(size_t)i * n_a + c];
  };
  // ---- |W|^2 in FP64, then the scaled columns in registers --------------------
  {
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < NC; ++s) {
      const int c = col_of(s);
#pragma unroll
      for (int e = 0; e < NV; ++e) {
        T x[VW];
#pragma unroll
        for (int q = 0; q < VW; ++q)
          x[q] = (c < l && row_of(e, q) < kw) ? Wat(row_of(e, q), c) : S<T>::zero();
#pragma unroll
        for (int q = 0; q < VW; ++q) acc += S<T>::abs2(x[q]);
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) sh.red64[warp] = acc;
    __syncthreads();
    if (tid < nc) {
      double t = 0.0;
      for (int w = 0; w < kCNW; ++w) t += sh.red64[w];
      cluster.map_shared_rank(&sh, tid)->p64[rank] = t;
    }
  }
  cluster.sync();
  double norm2 = 0.0;
  for (int r = 0; r < nc; ++r) norm2 += sh.p64[r];
  const double nrm = sqrt(norm2);
  const double scale = nrm > 0.0 ? 1.0 / nrm : 1.0;
  // stop once the trailing block holds at most max(thr_rel |W|^2, thr_abs)
  // (thr_rel < 0: only at an empty trailing block, so that all kmax rows come out)
  const float thr =
      thr_rel < 0.0 ? 0.f
                    : fmaxf((float)fmax(thr_rel, norm2 > 0.0 ? thr_abs / norm2 : 0.0), kQrFloor);
  F y[NC][NV * VW];
  int pst[NC];  // the step a column is the pivot of (INT_MAX: not yet; -1: no such column)
#pragma unroll
  for (int s = 0; s < NC; ++s) {
    const int c = col_of(s);
    pst[s] = c < l ? 0x7fffffff : -1;
#pragma unroll
    for (int e = 0; e < NV; ++e)
#pragma unroll
      for (int q = 0; q < VW; ++q) {
        const int i = row_of(e, q);
        y[s][e * VW + q] = (c < l && i < kw) ? F32<T>::from(Wat(i, c), scale) : F32<T>::zero();
      }
  }
  bool timeout = false;
  // Reflector of this warp's column s for pivot row j, v = x + nu e_j with
  // nu = (x_j/|x_j|)|x|, tau = 1/(|x|(|x|+|x_j|)), x_j <- -nu, x = rows j..: into slot
  // i of every CTA's ring; the column's rows below j become R's (zero).
  auto reflector = [&](F(&x)[NV * VW], int j, int i) {
    float n2 = 0.f;
    F xj = F32<T>::zero();
#pragma unroll
    for (int e = 0; e < NV; ++e) {
      if (VR * (e + 1) <= j) continue;
#pragma unroll
      for (int q = 0; q < VW; ++q) {
        const int row = row_of(e, q);
        if (row >= j) n2 += f_abs2(x[e * VW + q]);
        if (row == j) xj = x[e * VW + q];
      }
    }
    n2 = warp_sum(n2);
    xj = shfl_F(xj, (j / VW) & 31);
    const bool refl = n2 > kTinyCol * kTinyCol;
    const float xn = refl ? n2 * f_rsqrt(n2) : 0.f;
    float pr = 1.f, pi = 0.f, a0;  // phase and modulus of x_j
    if constexpr (sizeof(F) == 4) {
      pr = copysignf(1.f, xj);
      a0 = fabsf(xj);
    } else {
      const float x2 = f_abs2(xj);
      const float ia = x2 > 1e-36f ? f_rsqrt(x2) : 0.f;
      a0 = x2 * ia;
      if (ia > 0.f) {
        pr = re_F(xj) * ia;
        pi = im_F(xj) * ia;
      }
    }
    const float tau = refl ? f_rcp(xn * (xn + a0)) : 0.f;
    F v0, nu;
    set_F(v0, re_F(xj) + pr * xn, im_F(xj) + pi * xn);
    set_F(nu, -pr * xn, -pi * xn);
    // staged in this CTA's copy of the slot, then one bulk copy per CTA (lane d to CTA d)
    unsigned char* stage = ring_raw + (size_t)(kRing + i) * kSlot;
    float4* sv = reinterpret_cast<float4*>(stage + 16);
#pragma unroll
    for (int e = 0; e < NV; ++e) {
      if (VR * (e + 1) <= j) continue;
      F v[VW];
#pragma unroll
      for (int q = 0; q < VW; ++q) {
        const int row = row_of(e, q);
        F& z = x[e * VW + q];
        v[q] = row > j ? z : (row == j ? v0 : F32<T>::zero());
        if (row > j) z = F32<T>::zero();
        else if (row == j && refl) z = nu;
      }
      sv[lane + 32 * e] = vec_put(v);
    }
    if (lane == 0) *reinterpret_cast<float*>(stage) = tau;
    cl_bulk_fence();
    __syncwarp();
    if (lane < nc) {
      const uint32_t src = cl_smem(stage), dst = cl_map(cl_smem(ring_raw + (size_t)i * kSlot), lane);
      const uint32_t bar = cl_map(cl_smem(&sh.full[i]), lane), skip = (uint32_t)(j / VR) * 512u;
      if (skip) cl_bulk(dst, src, 16, bar);  // tau; otherwise one copy takes both
      cl_bulk(dst + (skip ? 16 + skip : 0), src + (skip ? 16 + skip : 0),
              NV * 512u - skip + (skip ? 0 : 16), bar);
    }
  };
  // This CTA's 8 heaviest columns into sh.mine, by counting; threads 128 ..
  auto rank_mine = [&]() {
    const int t = tid - 128;
    if (t >= 0 && t < kCNW * NC) {
      const int v = sh.cn[t];
      const int4* c4 = reinterpret_cast<const int4*>(sh.cn);
      int rk = 0;
#pragma unroll
      for (int u = 0; u < kCNW * NC / 4; ++u) {
        const int4 w = c4[u];
        rk += (w.x > v || (w.x == v && 4 * u < t)) + (w.y > v || (w.y == v && 4 * u + 1 < t)) +
              (w.z > v || (w.z == v && 4 * u + 2 < t)) + (w.w > v || (w.w == v && 4 * u + 3 < t));
      }
      if (rk < kRing) {
        const unsigned c = (unsigned)(rank * (kCNW * NC) + t);  // cn's index s 16 + warp is the column's
        sh.mine[rk] = (long long)(((unsigned long long)(unsigned)v << 32) | (0xffffffffu - c));
      }
    }
  };
  // the 8 heaviest of all CTAs, heaviest first: four threads count a candidate's betters
  auto select = [&](int par) {
    const int k = tid >> 2, q4 = tid & 3, n = nc * kRing;
    const longlong2* c2 = reinterpret_cast<const longlong2*>(sh.cand[par]);
    const long long v = k < n ? sh.cand[par][k] : 0;
    int rk = 0;
    for (int u = q4; u < n / 2; u += 4) {
      const longlong2 w = c2[u];
      rk += (w.x > v) + (w.y > v);
    }
    rk += __shfl_xor_sync(0xffffffffu, rk, 1);
    rk += __shfl_xor_sync(0xffffffffu, rk, 2);
    if (q4 == 0 && k < n && rk < kRing)
      sh.ord[rk] = v >= 0 ? (int)(0xffffffffu - (unsigned)v) : -1;
  };
  // thread (d, u): value u of this CTA to CTA d
  auto post_mine = [&](int par) {
    const int d = tid >> 3, u = tid & 7;
    if (d < nc) cluster.map_shared_rank(&sh, d)->cand[par][rank * kRing + u] = sh.mine[u];
  };
  auto key_of = [](float w) { return __float_as_int(w) & 0x7fffffff; };
  // first batch: the heaviest columns of W
  if (pivot) {
#pragma unroll
    for (int s = 0; s < NC; ++s) {
      float a = 0.f;
#pragma unroll
      for (int u = 0; u < NV * VW; ++u) a += f_abs2(y[s][u]);
      a = warp_sum(a);
      if (lane == 0) sh.cn[s * kCNW + warp] = pst[s] > 0 ? key_of(a) : -1;
    }
    __syncthreads();
    rank_mine();
    __syncthreads();
    if (tid < 128) post_mine(1);
    cluster.sync();
    select(1);
  }
  int keff = qsteps, level = 0;
  float trail = 0.f, before = 0.f;
  for (int b = 0; b * kRing < qsteps; ++b) {
    const int first = b * kRing, nb = min(kRing, qsteps - first), jl = first + nb - 1;
    const int par = b & 1;
    if (!pivot && tid < kRing) sh.ord[tid] = first + tid;
    __syncthreads();
    if (tid < nb) {  // the bytes of this batch's reflectors (whole vectors from the pivot's on)
      const int j = first + tid;
      cl_mbar_expect(&sh.full[tid], (uint32_t)((NV - j / VR) * 512 + 16));
    }
    {
      const int c0 = sh.ord[0];
#pragma unroll
      for (int s = 0; s < NC; ++s)
        if (pst[s] >= 0 && col_of(s) == c0) {
          pst[s] = first;
          reflector(y[s], first, 0);
        }
    }
    for (int i = 0; i < nb; ++i) {
      const int j = first + i;
      const int cnext = i + 1 < nb ? sh.ord[i + 1] : -1;
      if (!timeout && !cl_mbar_wait(&sh.full[i], par)) timeout = true;
      const unsigned char* slot = ring_raw + (size_t)i * kSlot;
      const float tau = *reinterpret_cast<const float*>(slot);
      const float4* vr = reinterpret_cast<const float4*>(slot + 16);
      F v[kKeep ? NV * VW : VW];  // the reflector, or one vector of it at a time
      float r0[NC], r1[NC], i0[NC], i1[NC];
#pragma unroll
      for (int s = 0; s < NC; ++s) r0[s] = r1[s] = i0[s] = i1[s] = 0.f;
#pragma unroll
      for (int e = 0; e < NV; ++e) {
        if (VR * (e + 1) <= j) continue;
        F* ve = &v[kKeep ? e * VW : 0];
        vec_get(vr[lane + 32 * e], ve);
#pragma unroll
        for (int s = 0; s < NC; ++s) {
#pragma unroll
          for (int q = 0; q < VW; ++q) {
            if (q & 1) f_dotc(ve[q], y[s][e * VW + q], r1[s], i1[s]);
            else f_dotc(ve[q], y[s][e * VW + q], r0[s], i0[s]);
          }
        }
      }
      float wr[NC], wi[NC];
#pragma unroll
      for (int s = 0; s < NC; ++s) {
        wr[s] = r0[s] + r1[s];
        wi[s] = i0[s] + i1[s];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int s = 0; s < NC; ++s) {
          wr[s] += __shfl_xor_sync(0xffffffffu, wr[s], o);
          if constexpr (sizeof(F) == 8) wi[s] += __shfl_xor_sync(0xffffffffu, wi[s], o);
        }
      }
#pragma unroll
      for (int e = 0; e < NV; ++e) {
        if (VR * (e + 1) <= j) continue;
        F* ve = &v[kKeep ? e * VW : 0];
        if constexpr (!kKeep) vec_get(vr[lane + 32 * e], ve);
#pragma unroll
        for (int s = 0; s < NC; ++s) {
          if (pst[s] <= j) continue;  // taken, or no column
#pragma unroll
          for (int q = 0; q < VW; ++q) f_axpy(tau * wr[s], tau * wi[s], ve[q], y[s][e * VW + q]);
        }
      }
#pragma unroll
      for (int s = 0; s < NC; ++s)
        if (pst[s] >= 0 && col_of(s) == cnext) {
          pst[s] = j + 1;
          reflector(y[s], j + 1, i + 1);
        }
    }
    // ---- weight below the batch, next pivots, stop test --------------------------
    float wtail = 0.f;
#pragma unroll
    for (int s = 0; s < NC; ++s) {
      float tail = 0.f;
      if (pst[s] > jl) {
#pragma unroll
        for (int e = 0; e < NV; ++e) {
          if (VR * (e + 1) <= jl) continue;
#pragma unroll
          for (int q = 0; q < VW; ++q)
            if (row_of(e, q) > jl) tail += f_abs2(y[s][e * VW + q]);
        }
      }
      tail = warp_sum(tail);
      wtail += tail;
      if (pivot && lane == 0) sh.cn[s * kCNW + warp] = pst[s] > jl ? key_of(tail) : -1;
    }
    if (lane == 0) sh.wsum[warp][0] = wtail;
    __syncthreads();
    if (tid < nc) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kCNW; ++w) t += sh.wsum[w][0];
      cluster.map_shared_rank(&sh, tid)->part[par][rank][0] = t;
    }
    if (pivot) {
      rank_mine();
      __syncthreads();
      if (tid < 128) post_mine(par);
    }
    cluster.sync();
    before = trail;
    trail = 0.f;
    for (int r = 0; r < nc; ++r) trail += sh.part[par][r][0];
    // A trailing block below kNoise whose weight 8 more pivots hardly reduce is the
    // rounding noise of FP32 around a matrix of lower rank (a spectrum that decays
    // towards the threshold falls faster): its rows hold nothing, and the Jacobi and
    // the FP64 products after it would take them along (337 rows for a rank of 258).
    if (plateau && trail > thr && trail < kNoise && trail > kFlat * before && b > 0) {
      keff = jl + 1;
      level = 1;
      break;
    }
    if (trail <= thr) {
      // the rank lies in this batch: the weight below each of its steps (the rows
      // between a step and the batch's last are R's and keep that weight)
      float acc[kRing];
#pragma unroll
      for (int u = 0; u < kRing; ++u) acc[u] = 0.f;
#pragma unroll
      for (int s = 0; s < NC; ++s)
#pragma unroll
        for (int e = 0; e < NV; ++e)
#pragma unroll
          for (int q = 0; q < VW; ++q) {
            const int row = row_of(e, q);
            const float a = f_abs2(y[s][e * VW + q]);
#pragma unroll
            for (int u = 0; u < kRing; ++u)
              if (row > first + u && pst[s] > first + u) acc[u] += a;
          }
#pragma unroll
      for (int u = 0; u < kRing; ++u) {
        acc[u] = warp_sum(acc[u]);
        if (lane == 0) sh.wsum[warp][u] = acc[u];
      }
      __syncthreads();
      if (tid < 128 && (tid >> 3) < nc) {
        float t = 0.f;
        for (int w = 0; w < kCNW; ++w) t += sh.wsum[w][tid & 7];
        cluster.map_shared_rank(&sh, tid >> 3)->part[par ^ 1][rank][tid & 7] = t;
      }
      cluster.sync();
      for (int u = 0; u < nb; ++u) {
        trail = 0.f;
        for (int r = 0; r < nc; ++r) trail += sh.part[par ^ 1][r][u];
        keff = first + u + 1;
        if (trail <= thr) break;
      }
      break;
    }
    if (pivot) {
      select(par);
      __syncthreads();
    }
  }
  // ---- R, column-major, columns in W's order ----------------------------------
#pragma unroll
  for (int s = 0; s < NC; ++s) {
    const int c = col_of(s);
    if (c >= l) continue;
    float4* out = reinterpret_cast<float4*>(Rg + (size_t)c * RP);
#pragma unroll
    for (int e = 0; e < NV; ++e) out[lane + 32 * e] = vec_put(&y[s][e * VW]);
  }
  if (timeout && lane == 0) atomicOr(&ctl_out->status, DEV_BARRIER_TIMEOUT);
  if (rank == 0 && tid == 0) {
    ctl_out->nact = keff;
    ctl_out->cap = qr_cap;
    ctl_out->plateau = level;
    ctl_out->pred = cap_dev ? cap_dev[1] : 0;
    info[0] = norm2;
    info[1] = (double)trail * norm2;
    info[5] = 1e-6 * (double)(global_ns() - t_start);
  }
  cluster.sync();  // no CTA leaves while another may still store into its shared memory
}

// vectors per lane for kw rows (0: too many)
template <typename T>
int nv_bucket(int kw) {
  constexpr bool real = sizeof(T) == sizeof(double);
  const int vr = real ? 128 : 64;
  const int need = (kw + vr - 1) / vr;
  for (int b : {1, 2, 4, 6, 8}) {
    if (need <= b) return b;
  }
  if (!real) {
    if (need <= 12) return 12;
    if (need <= 16) return 16;
  }
  return 0;
}
// CTAs for l columns: 16 warps each; a reflector goes to every CTA, so no more than
// the columns need
inline int qr_ctas(int l) { return l <= 4 * kCNW ? 4 : l <= 8 * kCNW ? 8 : kCWMax; }

// use(kernel, vectors per lane) with the kernel for kw rows and l columns; `none` beyond
// its sizes
template <typename T, typename Use, typename R>
R with_qr_kernel(int kw, int l, Use use, R none) {
  const int nc = qr_ctas(l), cols = (l + nc * kCNW - 1) / (nc * kCNW), nv = nv_bucket<T>(kw);
#define SM_QR(NVV, NCC) \
  if (nv == NVV && cols == NCC) return use(k_qr_cluster<T, NVV, NCC>, NVV)
  SM_QR(1, 1);
  SM_QR(1, 2);
  SM_QR(2, 1);
  SM_QR(2, 2);
  SM_QR(4, 1);
  SM_QR(4, 2);
  SM_QR(6, 1);
  SM_QR(6, 2);
  SM_QR(8, 1);
  SM_QR(8, 2);
  if constexpr (sizeof(T) == sizeof(double)) {
    SM_QR(1, 3);  // more than 512 columns have at most 512 rows
    SM_QR(2, 3);
    SM_QR(4, 3);
  } else {
    SM_QR(12, 1);
    SM_QR(12, 2);
    SM_QR(16, 1);
    SM_QR(16, 2);
  }
#undef SM_QR
  return none;
}
constexpr size_t qr_smem(int nv) { return (size_t)2 * kRing * (16 + nv * 512); }

}  // namespace

template <typename T>
int qr_row_pad(int kw) {
  return nv_bucket<T>(kw) * (sizeof(T) == sizeof(double) ? 128 : 64);
}

template <typename T>
bool qr_cluster_ok(Ctx& ctx, int kw, int l) {
  if (kw < 1 || l < 1 || kw > kMaxCol || std::min(kw, l) > kMaxRows ||
      l > (sizeof(T) == sizeof(double) ? 768 : 512))
    return false;
  return with_qr_kernel<T>(
      kw, l, [&](auto fn, int nv) { return cl_places(ctx, fn, qr_ctas(l), qr_smem(nv)); }, false);
}

template <typename T>
int qr_cluster(cudaStream_t st, const T* A, int n_a, int trans, int kw, int l, double thr_rel,
               double thr_abs, typename F32<T>::type* Rg, JacobiCtl* ctl, double* info, int qr_cap,
               const int* cap_dev, int pivot, int plateau) {
  const int rc = with_qr_kernel<T>(
      kw, l,
      [&](auto fn, int nv) {
        return cl_launch(fn, qr_ctas(l), qr_smem(nv), st, A, n_a, trans, kw, l, thr_rel, thr_abs, Rg,
                         ctl, info, qr_cap, cap_dev, pivot, plateau);
      },
      (int)SM_ERR_VALUE);
  if (rc == SM_ERR_VALUE) set_error("mixed split: matrix beyond the cluster QR's limits");
  return rc;
}

template int qr_row_pad<double>(int);
template int qr_row_pad<cplx>(int);
template bool qr_cluster_ok<double>(Ctx&, int, int);
template bool qr_cluster_ok<cplx>(Ctx&, int, int);
template int qr_cluster<double>(cudaStream_t, const double*, int, int, int, int, double, double,
                                float*, JacobiCtl*, double*, int, const int*, int, int);
template int qr_cluster<cplx>(cudaStream_t, const cplx*, int, int, int, int, double, double, float2*,
                              JacobiCtl*, double*, int, const int*, int, int);

}  // namespace sm
