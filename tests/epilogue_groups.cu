// The two accumulators of gemm_pair_kernel on the host: barriers with the parity rule of an mbarrier, an MMA thread that works on, the epilogue
// warps of both groups and both blocks.  Prints, for every instance, how often a warp took another tile's accumulator for its own, or waited for
// one that never came: with the arrivals the kernel counts (TileCfg::kHandBacks), and with the first group's alone.
#include <cstdio>
#include <random>

#include "gemm_tcgen05_pair.cuh"

namespace {

struct Barrier {
  int arrivals = 0, phases = 0;
  void arrive(int count) {
    if (++arrivals == count) arrivals = 0, ++phases;
  }
  bool passes(unsigned int parity) const { return (static_cast<unsigned int>(phases) & 1u) != parity; }
};

// One step of the model is one event of an actor chosen at random: the MMA thread completes a tile, a warp passes its wait or ends its
// epilogue.  `late`: that one warp moves only once in so many times.
template <int GROUPS, int CTAS>
int mistakes(int hand_backs, unsigned int seed, int late) {
  constexpr int WARPS = 4 * GROUPS * CTAS, TILES = 7;
  const bool second_arrives = hand_backs == WARPS;
  std::mt19937 rng(seed);
  Barrier full[2], empty[2];
  int next[WARPS] = {}, issued = 0, wrong = 0, idle = 0, left = WARPS;
  bool working[WARPS] = {};
  const int slow = static_cast<int>(rng() % WARPS);
  while (left > 0 && wrong == 0) {
    const int actor = static_cast<int>(rng() % (WARPS + 1));
    bool moved = false;
    if (actor == WARPS) {
      if (issued < TILES && empty[issued & 1].passes((issued >> 1 & 1u) ^ 1u)) {
        full[issued & 1].arrive(1);
        ++issued;
        moved = true;
      }
    } else if (next[actor] < TILES && !(actor == slow && rng() % late)) {
      const int n = next[actor], acc = n & 1;
      const bool second = GROUPS == 2 && actor / 4 % 2 == 1, last = n == TILES - 1;
      bool through = false;
      if (!working[actor] && full[acc].passes(n >> 1 & 1u)) {
        wrong += full[acc].phases != (n >> 1) + 1;
        working[actor] = moved = true;
        through = second && !last;
      } else if (working[actor]) {
        through = true;
      }
      if (through) {
        if (!last && (!second || second_arrives)) empty[acc].arrive(hand_backs);
        working[actor] = false;
        left -= ++next[actor] == TILES;
        moved = true;
      }
    }
    idle = moved ? 0 : idle + 1;
    if (idle > 100000) return 1;  // nothing can happen any more: a wait for a phase that does not come
  }
  return wrong;
}

template <int MODE, int SRC, int BN, int CTAS>
void report() {
  using Cfg = sb200::TileCfg<MODE, SRC, BN, CTAS>;
  constexpr int GROUPS = Cfg::kEpiGroups;
  int counts[2] = {0, 0};
  for (unsigned int seed = 0; seed < 500; ++seed) {
    const int late = 1 + static_cast<int>(seed % 100);
    counts[0] += mistakes<GROUPS, CTAS>(Cfg::kHandBacks, seed, late);
    counts[1] += mistakes<GROUPS, CTAS>(4 * CTAS, seed, late);
  }
  std::printf("%d %d %d %d groups=%d mistakes=%d first=%d\n", MODE, SRC, BN, CTAS, GROUPS, counts[0], counts[1]);
}

template <int MODE, int SRC>
void widths() {
  report<MODE, SRC, 64, 1>();
  report<MODE, SRC, 128, 1>();
  report<MODE, SRC, 64, 2>();
  report<MODE, SRC, 128, 2>();
  report<MODE, SRC, 192, 2>();
  report<MODE, SRC, 256, 2>();
}

}  // namespace

int main() {
  widths<1, sb200::SRC_DIRECT>();
  widths<3, sb200::SRC_DIRECT>();
  widths<3, sb200::SRC_PANELS>();
  widths<2, sb200::SRC_PANELS>();
  widths<4, sb200::SRC_PANELS>();
  report<5, sb200::SRC_DIRECT, 256, 2>();
}
