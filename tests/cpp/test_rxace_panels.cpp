// Host only: the plain RX/ACE scorer's schedule, for every band and target count.
// Each pair of row groups belongs to one warp, the groups' weights lie apart on
// 16-byte offsets, and the warps, each taking its pairs in order and waiting for
// the pair eight before, all come to the end.
#include "../../hsi-detectors-cuda_b200/csrc/rxace_panels.h"

#include <set>
#include <string>

#include "check.hpp"

using namespace hsi_b200;

namespace {

bool every_warp_finishes(const Panels& p, int pairs) {
  int at[kSimtWarps];
  for (int w = 0; w < kSimtWarps; ++w) at[w] = p.first[w];
  std::vector<bool> done(pairs, false);
  for (bool moved = true; moved;) {
    moved = false;
    for (int w = 0; w < kSimtWarps; ++w) {
      if (at[w] == p.first[w + 1]) continue;
      const int pair = p.pair[at[w]];
      if (pair >= kChains / 2 && !done[pair - kChains / 2]) continue;  // waits
      done[pair] = true;
      ++at[w];
      moved = true;
    }
  }
  for (int w = 0; w < kSimtWarps; ++w)
    if (at[w] != p.first[w + 1]) return false;
  return true;
}

}  // namespace

int main() {
  for (int B = 1; B <= HSI_MAX_BANDS; ++B)
    for (int T = 0; T <= HSI_MAX_FILTERS_PER_PASS; ++T) {
      const Panels p = make_panels(B, T);
      const std::string at = "B " + std::to_string(B) + " T " + std::to_string(T);
      auto check = [&](bool ok, const char* what) { tcheck::report(ok, what, __FILE__, __LINE__, at); };
      const int pairs = (p.groups + 1) / 2;
      check(p.groups <= kMaxGroups && p.groups * kGroupRows >= B + T && p.kpad % kGroupRows == 0 && p.kpad >= B, "sizes");
      check(p.first[0] == 0 && p.first[kSimtWarps] == pairs, "as many list entries as pairs");
      std::set<int> seen;
      bool ascending = true;
      for (int w = 0; w < kSimtWarps; ++w)
        for (int i = p.first[w]; i < p.first[w + 1]; ++i) {
          seen.insert(p.pair[i]);
          if (i > p.first[w] && p.pair[i] <= p.pair[i - 1]) ascending = false;
        }
      check(static_cast<int>(seen.size()) == pairs && *seen.begin() == 0 && *seen.rbegin() == pairs - 1, "each pair once");
      check(ascending, "a warp's pairs ascend");
      check(every_warp_finishes(p, pairs), "no warp waits for ever");
      std::vector<bool> used(p.floats, false);
      bool apart = true;
      for (int g = 0; g < p.groups; ++g) {
        check(p.offset[g] % 4 == 0 && p.bands[g] % 8 == 0 && p.bands[g] <= p.kpad, "alignment");
        check(p.bands[g] >= (g * kGroupRows < B ? std::min((g + 1) * kGroupRows, B) : B), "rows reach their last band");
        for (int i = 0; i < p.bands[g] * kGroupRows; ++i) {
          const int f = p.offset[g] + i;
          if (f >= p.floats || used[f]) apart = false;
          else used[f] = true;
        }
      }
      check(apart, "panels lie apart");
    }
  return tcheck::finish("rxace_panels");
}
