// How products are cut for the SMs of the device: plain host functions of sizes and SM
// count (tests/test_tile_rules.py).
#pragma once

#include <cmath>

namespace sm {

// FP64 GEMM (k_gemm): the tile (16 or 32) and the number of K slices whose fullest SM
// has the least to do: a CTA takes tile^2 kchunk / 2 clocks of its SM's FP64 pipe
// (complex four times that) and some 1500 clocks of loads and stores that only further
// CTAs hide, the slices' sum as much again.  (130 x 130 x 256 on 152 SMs: 25 tiles of
// 32 in 6 slices, 150 CTAs, against 8 slices, 200 CTAs: 22 us.)
struct GemmCut {
  int tile, slices;
};
inline double gemm_cost(int M, int N, int K, bool cplx, int sms, GemmCut c) {
  const double tiles = (double)((M + c.tile - 1) / c.tile) * ((N + c.tile - 1) / c.tile);
  const int kc = ((K + c.slices - 1) / c.slices + 15) / 16 * 16;
  const double cta = 0.5 * c.tile * c.tile * kc * (cplx ? 4.0 : 1.0) + 1500.0;
  return std::ceil(tiles * c.slices / sms) * cta + (c.slices > 1 ? 1500.0 : 0.0);
}
inline GemmCut gemm_cut(int M, int N, int K, bool cplx, int sms) {
  GemmCut best = {16, 1};
  double cost = gemm_cost(M, N, K, cplx, sms, best);
  for (int t = 16; t <= 32; t += 16)
    for (int nz = 1; nz <= 8 && (nz == 1 || K > 16 * (nz - 1)); ++nz) {
      const double c = gemm_cost(M, N, K, cplx, sms, {t, nz});
      if (c < cost) {
        cost = c;
        best = {t, nz};
      }
    }
  return best;
}

// FP32 products of the rank predictor (k_sgemm): K slices of at least one slab of `slab`,
// a power of two up to 8, until there are two CTAs per SM.
inline int sgemm_slices(long tiles, int K, int slab, int sms) {
  int nz = 1;
  while (nz < 8 && tiles * nz < 2L * sms && K > slab * nz) nz *= 2;
  return nz;
}

}  // namespace sm
