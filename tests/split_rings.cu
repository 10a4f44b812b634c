// The rings of gemm_split_kernel on the host: barriers with the parity rule of an mbarrier, loads that land in any order, the kernel's own
// waits (split_waits).  Prints, for every instance, how many waits for a raw stage passed before their k-block had landed: in the kernel's
// order of the two waits, and in the other one.
#include <cstdio>
#include <random>

#include "gemm_split.cuh"

namespace {

struct Barrier {
  int arrivals = 0, phases = 0;
  void arrive(int count) {
    if (++arrivals == count) arrivals = 0, ++phases;
  }
  bool passes(unsigned int parity) const { return (static_cast<unsigned int>(phases) & 1u) != parity; }
};

// One step of the model is one event of an actor chosen at random: a load lands, a group passes its waits or ends its k-block, the
// tensor core takes one.  `late`: one k-block in so many lands only when little else can happen.
template <class Cfg, int CTAS>
int early_passes(bool kernel_order, unsigned int seed, int late) {
  constexpr int RAW = Cfg::kRaw, PARTS = Cfg::kParts, GROUPS = Cfg::kGroups, BLOCKS = 60;
  std::mt19937 rng(seed);
  Barrier raw_full[CTAS][RAW], raw_empty[CTAS][RAW], part_full[PARTS], part_empty[PARTS];
  bool landed[CTAS][BLOCKS] = {}, slow[CTAS][BLOCKS], working[CTAS][GROUPS] = {};
  int issued[CTAS] = {}, next[CTAS][GROUPS], multiplied = 0, early = 0, idle = 0;
  for (int c = 0; c < CTAS; ++c) {
    for (int n = 0; n < BLOCKS; ++n) slow[c][n] = rng() % late == 0;
    for (int g = 0; g < GROUPS; ++g) next[c][g] = g;
  }
  while (multiplied < BLOCKS && early == 0) {
    const int c = static_cast<int>(rng() % CTAS), actor = static_cast<int>(rng() % (GROUPS + 3));
    bool moved = false;
    if (actor < GROUPS) {
      const int g = actor;
      const unsigned int n = static_cast<unsigned int>(next[c][g]);
      if (n >= BLOCKS) continue;
      if (!working[c][g]) {
        auto part = [&](unsigned int stage, unsigned int parity) { return part_empty[stage].passes(parity); };
        auto raw = [&](unsigned int stage, unsigned int parity) { return raw_full[c][stage].passes(parity); };
        // the other order: the raw stage is waited for, and read, at a moment when the part stage may still be taken
        if (kernel_order ? sb200::split_waits<Cfg>(n, part, raw) : raw(n % RAW, n / RAW & 1u)) {
          early += !landed[c][n];
          working[c][g] = moved = true;
        }
      } else if (part_empty[n % PARTS].passes((n / PARTS & 1u) ^ 1u)) {
        raw_empty[c][n % RAW].arrive(1);
        part_full[n % PARTS].arrive(CTAS);
        working[c][g] = false;
        next[c][g] += GROUPS;
        moved = true;
      }
    } else if (actor == GROUPS) {
      const int n = issued[c];
      if (n < BLOCKS && raw_empty[c][n % RAW].passes((n / RAW & 1u) ^ 1u)) {
        ++issued[c];
        moved = true;
      }
    } else if (actor == GROUPS + 1) {
      const int n = issued[c] - 1 - static_cast<int>(rng() % RAW);
      if (n >= 0 && !landed[c][n] && (!slow[c][n] || idle > 200)) {
        landed[c][n] = moved = true;
        raw_full[c][n % RAW].arrive(1);
      }
    } else if (part_full[multiplied % PARTS].passes(multiplied / PARTS & 1)) {
      part_empty[multiplied % PARTS].arrive(1);
      ++multiplied;
      moved = true;
    }
    idle = moved ? 0 : idle + 1;
    if (idle > 100000) return -1;  // nothing can happen any more
  }
  return early;
}

template <int BN, int CTAS, int ROWS>
void report() {
  using Cfg = sb200::SplitCfg<BN, CTAS, ROWS>;
  int counts[2] = {0, 0};
  for (int order = 0; order < 2; ++order)
    for (unsigned int seed = 0; seed < 2000; ++seed) {
      const int e = early_passes<Cfg, CTAS>(order == 0, seed, 3 + static_cast<int>(seed % 20));
      counts[order] = e < 0 || counts[order] < 0 ? -1 : counts[order] + e;
    }
  std::printf("%d %d %d raw=%d parts=%d groups=%d early=%d other=%d\n", BN, CTAS, ROWS, Cfg::kRaw, Cfg::kParts, Cfg::kGroups, counts[0], counts[1]);
}

}  // namespace

int main() {
  report<64, 1, 64>();
  report<128, 1, 64>();
  report<64, 1, 128>();
  report<128, 1, 128>();
  report<64, 2, 128>();
  report<128, 2, 128>();
  report<192, 2, 128>();
  report<256, 2, 128>();
}
