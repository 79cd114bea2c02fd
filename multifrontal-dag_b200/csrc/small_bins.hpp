// Size bins of the small fronts: which launch of its level a front goes to (host).
#pragma once
#include <algorithm>
#include <vector>

#include "plan.hpp"

namespace mfd {

constexpr int kWarpFrontsAtOnce = kNumSms * 24;   // one-warp fronts the chip holds at once

// The bins' largest orders, ascending, of a handle whose small fronts have at most sfm rows.
inline std::vector<int> small_bin_sizes(int sfm) {
  std::vector<int> bins{16, 24, 32, 64, 96, 128, 160};
  while (!bins.empty() && bins.back() > sfm) bins.pop_back();
  if (bins.empty() || bins.back() < sfm) bins.push_back(sfm);
  return bins;
}

// The bin of every front of a level, given their orders; -1: above sfm, a large front.
// The one-warp fronts (of at most 32 rows and on this side of the line) go to one launch sized for
// the largest unless they fill the chip more than once: below that the launches' number counts,
// not their warps' registers and shared memory.
inline std::vector<int> small_bins_of_level(const std::vector<int>& bins, int sfm, const std::vector<int>& orders) {
  const int warp_line = std::min(32, sfm);
  int warp_fronts = 0, warp_max = 0;
  for (int nf : orders) {
    if (nf > warp_line) continue;
    ++warp_fronts;
    warp_max = std::max(warp_max, nf);
  }
  const bool split = warp_fronts > kWarpFrontsAtOnce;
  std::vector<int> of;
  of.reserve(orders.size());
  for (int nf : orders) {
    int b = -1;
    if (nf <= sfm) {
      const int fit = nf <= warp_line && !split ? warp_max : nf;
      b = (int)(std::lower_bound(bins.begin(), bins.end(), fit) - bins.begin());
    }
    of.push_back(b);
  }
  return of;
}

}  // namespace mfd
