// rxace_panels.h - how the plain RX/ACE scorer (rxace.cu) shares its rows among
// the warps of a block: host code, so that the schedule can be checked without a
// device.
#pragma once

#include <algorithm>

#include "hsi_b200.h"

namespace hsi_b200 {

constexpr int kSimtWarps = 8;
constexpr int kGroupRows = 8;   // output rows (bands + targets) per group
constexpr int kChains = 16;     // partial sums of RX per pixel: groups G, G + 16, G + 32 each
constexpr int kMaxGroups = (HSI_MAX_BANDS + HSI_MAX_FILTERS_PER_PASS) / kGroupRows;
constexpr int kMaxPairs = (kMaxGroups + 1) / 2;

// Where the groups' weights lie (floats from the panels' start, [k][8 rows] of
// `bands[g]` bands) and which warp takes which pairs of groups (2 i, 2 i + 1).
struct Panels {
  int groups;
  int kpad;                       // bands rounded up to 8
  int floats;                     // of all panels
  int offset[kMaxGroups];
  short bands[kMaxGroups];
  unsigned char first[kSimtWarps + 1];  // warp w's pairs: pair[first[w]] .. pair[first[w + 1] - 1], ascending
  unsigned char pair[kMaxPairs];
};

constexpr int round_up(int v, int m) { return (v + m - 1) / m * m; }

// A pair waits for the pair kChains / 2 before it, so a warp's pairs ascend: the
// lowest unfinished pair of a block is always at the head of its warp's list and
// waits for nothing unfinished.
inline Panels make_panels(int B, int T) {
  Panels p{};
  p.groups = (B + T + kGroupRows - 1) / kGroupRows;
  p.kpad = round_up(B, kGroupRows);
  const int pairs = (p.groups + 1) / 2;
  for (int g = 0; g < p.groups; ++g)  // rows above B end their dot product at the diagonal; target rows are dense
    p.bands[g] = static_cast<short>(std::min((g + 1) * kGroupRows, p.kpad));
  // longest pair first, each to the warp with the least to do
  int load[kSimtWarps] = {}, warp_of[kMaxPairs];
  for (int i = pairs - 1; i >= 0; --i) {
    const int w = static_cast<int>(std::min_element(load, load + kSimtWarps) - load);
    warp_of[i] = w;
    load[w] += p.bands[std::min(2 * i + 1, p.groups - 1)];
  }
  int n = 0;
  for (int w = 0; w < kSimtWarps; ++w) {
    p.first[w] = static_cast<unsigned char>(n);
    for (int i = 0; i < pairs; ++i)
      if (warp_of[i] == w) p.pair[n++] = static_cast<unsigned char>(i);
  }
  p.first[kSimtWarps] = static_cast<unsigned char>(n);
  // the two halves of a warp read their weights at the same band: the odd
  // groups' panels start 64 bytes off, on other banks
  for (int half = 0; half < 2; ++half) {
    if (half) p.floats += 16;
    for (int g = half; g < p.groups; g += 2) {
      p.offset[g] = p.floats;
      p.floats += p.bands[g] * kGroupRows;
    }
  }
  return p;
}

}  // namespace hsi_b200
