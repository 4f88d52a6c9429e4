// Replays the dense lists of walk groups whose traversals pause, with every
// dense job reading as late as it can: after its group's own job has written
// what follows the pause.  A dense job must read the cells that were published
// to it, never what came later (a run of particles in a cell's place is a
// particle index taken for a node).  Prints "ok" or the first wrong read.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "bhg_lists.h"

struct Entry {
  uint32_t group, leg;
};

int main() {
  const size_t cap = 64, cells = 40;
  for (size_t warps : {4, 8, 100, 2368, 3552}) {
    for (size_t ngroups : {(size_t)1, warps / 4, warps / 2}) {
      std::vector<Entry> lists(warps * cap, Entry{~0u, ~0u});
      for (uint32_t leg = 0; leg < 3; ++leg)  // a traversal that pauses twice
        for (size_t gi = 0; gi < ngroups; ++gi) {
          const size_t slot = bhg::dense_slot(true, leg > 0, gi, ngroups, gi);
          if (slot >= warps) return std::printf("list %zu of %zu\n", slot, warps), 1;
          for (size_t i = 0; i < (leg ? cap : cells); ++i) lists[slot * cap + i] = Entry{(uint32_t)gi, leg};
        }
      for (size_t gi = 0; gi < ngroups; ++gi) {
        const size_t slot = bhg::dense_slot(true, false, gi, ngroups, ngroups + gi);
        for (size_t i = 0; i < cells; ++i) {
          const Entry e = lists[slot * cap + i];
          if (e.group != gi || e.leg != 0)
            return std::printf("%zu groups: dense job %zu reads leg %u of group %u\n", ngroups, gi, e.leg, e.group), 1;
        }
      }
    }
    for (size_t w = 0; w < warps; ++w)  // without dense jobs: the warp's own
      if (bhg::dense_slot(false, w & 1, 0, 1, w) != w) return std::printf("warp %zu\n", w), 1;
  }
  std::printf("ok\n");
  return 0;
}
