// Division of a scratch pool among simulations that can use more than they
// need.  Plain C++, so that it can be checked without a device.
#pragma once

#include <stddef.h>

#include <vector>

namespace nb {

// Units for each of several simulations, of which i runs with least[i] and has
// no use for more than whole[i]: the least for all (whether or not `total` holds
// it), and of what is left of `total` as large a part as of everybody's wish.
inline std::vector<size_t> share_scratch(const std::vector<size_t>& least,
                                         const std::vector<size_t>& whole, size_t total) {
  size_t low = 0, high = 0;
  for (size_t i = 0; i < least.size(); ++i) {
    low += least[i];
    high += whole[i];
  }
  if (high <= total) return whole;
  std::vector<size_t> got = least;
  if (low < total)
    for (size_t i = 0; i < got.size(); ++i)
      got[i] += (size_t)((unsigned __int128)(whole[i] - least[i]) * (total - low) / (high - low));
  return got;
}

}  // namespace nb
