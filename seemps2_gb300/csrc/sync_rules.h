// Who writes where, and when, in the kernels whose CTAs exchange data without a barrier
// around every access: plain functions that the kernels use and a host test runs every
// order of events through (tests/test_sync_rules.py).
#pragma once

#ifdef __CUDACC__
#define SM_RULE __host__ __device__ constexpr
#else
#define SM_RULE constexpr
#endif

namespace sm {

// ---- k_jacobi_cluster: the block rounds ------------------------------------------
// CTA c of nc holds a top (0) and a bottom (1) block. After a round the tops move one
// CTA up and the bottoms one CTA down; CTA 0's top stays, its bottom becomes CTA 1's
// top, and the last CTA's top becomes its own bottom.
struct JacBlock {
  int cta, half;
};
SM_RULE JacBlock jac_dest(int c, int half, int nc) {
  if (half) return c > 0 ? JacBlock{c - 1, 1} : JacBlock{1, 0};
  return c == 0 ? JacBlock{0, 0} : c + 1 == nc ? JacBlock{c, 1} : JacBlock{c + 1, 0};
}
// where the block that CTA c gets as its top or bottom comes from
SM_RULE JacBlock jac_source(int c, int half, int nc) {
  if (half) return c + 1 == nc ? JacBlock{c, 0} : JacBlock{c + 1, 1};
  return c == 0 ? JacBlock{0, 0} : c == 1 ? JacBlock{0, 1} : JacBlock{c - 1, 0};
}
// A block is copied out of its round's buffer, and one round later the CTA that fills
// the buffer's place in the next order writes over it. That CTA need not be the one
// that received the copy, so the receiver tells it: the CTA to which c, once it has
// its rows of a round, reports those of its `half` (-1: no report is needed, because
// the rows never left the CTA or c itself is the next to write there).
SM_RULE int jac_report(int c, int half, int nc) {
  const JacBlock s = jac_source(c, half, nc);
  if (s.cta == c) return -1;
  const int writer = jac_source(s.cta, s.half, nc).cta;
  return writer == c ? -1 : writer;
}
// reports that CTA c waits for before it sends the next round's rows
SM_RULE int jac_reports(int c, int nc) {
  int n = 0;
  for (int k = 0; k < nc; ++k)
    for (int half = 0; half < 2; ++half) n += jac_report(k, half, nc) == c;
  return n;
}

// ---- k_house_qr, k_house_qr_reg: sums over the grid --------------------------------
// Each CTA leaves its part of a sum before a step's grid barrier and all CTAs read the
// parts after it, while the fastest of them may already be in the next step: what a
// step writes before its barrier must not be what the step before it reads after its
// own.  Slots (a part per CTA each) by step j:
// the streaming kernel sums once a step; |W|^2, summed before step 0, is in slot 0
SM_RULE int qr_step_slot(int j) { return (j + 1) & 1; }
constexpr int kQrStepSlots = 2;
// the register kernel sums once per kQrBatch steps, for each of them, and a last batch
// may be a single step; |W|^2 has the slot after the two batches'
constexpr int kQrBatch = 4;
SM_RULE int qr_batch_slot(int j) { return j / kQrBatch % 2 * kQrBatch; }
constexpr int kQrNormSlot = 2 * kQrBatch, kQrBatchSlots = 2 * kQrBatch + 1;
static_assert(kQrStepSlots <= kQrBatchSlots, "one buffer serves both");

}  // namespace sm
