// Runs the rules of csrc/sync_rules.h through random orders of events; prints "ok" or
// what went wrong. "jacobi-outs" sends from buffers apart instead of
// reporting, "jacobi-blind" does neither, "qr-step-single" and
// "qr-batch-single" keep one buffer for the sums.
#include <cstdio>
#include <cstring>
#include <map>
#include <random>
#include <tuple>
#include <vector>

#include "sync_rules.h"

using namespace sm;

namespace {

// An mbarrier: a phase ends when its arrivals and its bytes are in.
struct Bar {
  int count = 1, pending = 1, tx = 0;
  long phase = 0;
  void init(int n) { count = pending = n; }
  void close() {
    if (pending == 0 && tx == 0) {
      ++phase;
      pending = count;
    }
  }
  void arrive() {
    --pending;
    close();
  }
  void expect(int n) {
    tx += n;
    arrive();
  }
  void complete() {
    --tx;
    close();
  }
  bool done(int parity) const { return (phase & 1) != parity; }
};

struct Copy {
  int src, src_half, dst, dst_half, par;  // par: of the source; the other of the destination
};

// The block rounds of k_jacobi_cluster, one row to a block: every CTA's steps in order,
// the copies delivered whenever the order of events likes.
// `outs`: the copies leave from buffers of their own, two to a block, and nothing is
// reported. Else the reports are made by a warp of its own (`apart`) or last in a round.
const char* jacobi(int nc, int rounds, bool reports, bool outs, bool apart, unsigned seed) {
  std::mt19937 rng(seed);
  struct Cta {
    int g = 0, step = 0, told = 0;
    Bar bar[2], clear[2];
  };
  std::vector<Cta> c(nc);
  for (int k = 0; k < nc; ++k)
    for (int p = 0; p < 2; ++p) c[k].clear[p].init(jac_reports(k, nc) > 0 ? jac_reports(k, nc) : 1);
  // [half][cta][parity]: which block lies there
  std::vector<std::vector<std::vector<int>>> block(2);
  for (int h = 0; h < 2; ++h)
    for (int k = 0; k < nc; ++k) block[h].push_back({h ? 2 * nc - 1 - k : k, -1});
  auto sent = block;  // the buffers apart
  std::vector<Copy> flight;
  std::vector<int> met(4 * nc * nc, 0);
  const bool slow = rng() % 2;  // prefer the CTAs over the copies
  while (true) {
    std::vector<int> can;
    for (int k = 0; k < nc; ++k) {
      const Cta& x = c[k];
      const bool duty = jac_report(k, 0, nc) >= 0 || jac_report(k, 1, nc) >= 0;
      if (apart && duty && x.told < rounds && x.bar[x.told & 1].done((x.told >> 1) & 1))
        can.push_back(nc + k);
      if (x.g == rounds) continue;
      const int ap = x.g & 1;
      bool on = true;
      if (x.step == 1 && reports && jac_reports(k, nc) > 0 && x.g > 0)
        on = x.clear[ap ^ 1].done(((x.g - 1) >> 1) & 1);
      if (x.step == 3) on = x.bar[ap].done((x.g >> 1) & 1);
      if (on) can.push_back(k);
    }
    if (can.empty() && flight.empty()) break;
    const bool deliver = can.empty() || (!flight.empty() && rng() % (slow ? 40 : 2) == 0);
    if (deliver) {
      const size_t i = rng() % flight.size();
      const Copy f = flight[i];
      flight.erase(flight.begin() + i);
      block[f.dst_half][f.dst][f.par ^ 1] = (outs ? sent : block)[f.src_half][f.src][f.par];
      c[f.dst].bar[f.par].complete();
      continue;
    }
    const int actor = can[rng() % can.size()], k = actor % nc;
    Cta& x = c[k];
    const int round = actor < nc ? x.g : x.told;
    if (actor >= nc || (!apart && x.step == 3))
      for (int h = 0; h < 2; ++h) {
        const int to = jac_report(k, h, nc);
        if (to >= 0) c[to].clear[round & 1].arrive();
      }
    if (actor >= nc) {
      ++x.told;
      continue;
    }
    const int ap = x.g & 1, np = ap ^ 1;
    if (x.step == 0) {  // the round's pairs
      int in = 0;
      for (int h = 0; h < 2; ++h) in += jac_source(k, h, nc).cta != k;
      x.bar[ap].expect(in);
      const int a = block[0][k][ap], b = block[1][k][ap];
      if (a < 0 || b < 0 || a == b) return "a CTA without two blocks";
      ++met[a * 2 * nc + b];
      ++met[b * 2 * nc + a];
    } else if (x.step == 2) {  // both blocks on their way
      for (int h = 0; h < 2; ++h) {
        const JacBlock d = jac_dest(k, h, nc);
        const JacBlock s = jac_source(d.cta, d.half, nc);
        if (s.cta != k || s.half != h) return "jac_source does not undo jac_dest";
        for (const Copy& f : flight)
          if (outs ? f.src == k && f.src_half == h && f.par == ap
                   : f.src == d.cta && f.src_half == d.half && f.par == np)
            return "a write over the source of a copy in flight";
        sent[h][k][ap] = block[h][k][ap];
        // its CTA is done with it once it has sent the rows of the round before
        const Cta& y = c[d.cta];
        if (d.cta != k && (y.g < x.g - 1 || (y.g == x.g - 1 && y.step < 3)))
          return "a write into a buffer in use";
        if (d.cta == k) block[d.half][k][np] = block[h][k][ap];
        else flight.push_back({k, h, d.cta, d.half, ap});
      }
    }
    if (++x.step == 4) {
      x.step = 0;
      ++x.g;
    }
  }
  for (int k = 0; k < nc; ++k) {
    const bool duty = jac_report(k, 0, nc) >= 0 || jac_report(k, 1, nc) >= 0;
    if (c[k].g != rounds || (apart && duty && c[k].told != rounds)) return "a wait that does not end";
  }
  const int sweeps = rounds / (2 * nc - 1);
  for (int a = 0; a < 2 * nc; ++a)
    for (int b = 0; b < 2 * nc; ++b)
      if (a != b && met[a * 2 * nc + b] != sweeps) return "blocks that do not meet once a sweep";
  return nullptr;
}

// The grid sums of the Householder QR: between two grid barriers some CTAs read the sums
// published before the first while others publish those of the second.  Barrier 0 follows
// |W|^2, barrier j + 1 step j.
const char* qr_sums(int nmax, bool batches, bool alternate) {
  auto slots = [&](int b) {  // published before barrier b
    std::vector<int> s;
    if (b == 0) {
      s.push_back(!batches ? 0 : alternate ? kQrNormSlot : kQrBatch - 1);
    } else if (!batches) {
      s.push_back(alternate ? qr_step_slot(b - 1) : 0);
    } else {
      const int j = b - 1, n = j % kQrBatch + 1;
      if (n == kQrBatch || j + 1 == nmax)
        for (int i = 0; i < n; ++i) s.push_back((alternate ? qr_batch_slot(j) : 0) + i);
    }
    return s;
  };
  for (int b = 0; b < nmax; ++b)
    for (int read : slots(b)) {
      if (read < 0 || read >= (batches ? kQrBatchSlots : kQrStepSlots)) return "a slot out of range";
      for (int write : slots(b + 1))
        if (read == write) return "a sum written over while it is read";
    }
  return nullptr;
}

}  // namespace

int main(int argc, char** argv) {
  const char* mode = argc > 1 ? argv[1] : "";
  if (!std::strncmp(mode, "jacobi", 6)) {
    const bool outs = !std::strcmp(mode, "jacobi-outs"), reports = !std::strcmp(mode, "jacobi");
    for (int nc = 2; nc <= 16; ++nc)
      for (unsigned seed = 0; seed < 120; ++seed)
        if (const char* bad = jacobi(nc, 3 * (2 * nc - 1), reports, outs, reports && seed % 2, seed)) {
          std::printf("%d CTAs: %s\n", nc, bad);
          return 0;
        }
  }
  if (!std::strncmp(mode, "qr", 2)) {
    const bool batches = std::strstr(mode, "batch"), alternate = !std::strstr(mode, "single");
    for (int nmax = 1; nmax <= 64; ++nmax)
      if (const char* bad = qr_sums(nmax, batches, alternate)) {
        std::printf("%d steps: %s\n", nmax, bad);
        return 0;
      }
  }
  std::printf("ok\n");
  return 0;
}
