// Sizes of the tree build's levels: which leaf groups a tree of n particles
// starts from and how much room a workspace needs for them.  Plain C++, so that
// the bounds can be checked over all sizes without a device.
#pragma once

#include <stddef.h>

namespace nb {

constexpr int kLevelItems = 2048;      // capacity of a later level's CTA

// Open splits a CTA hands on at most: 2 x depth + 1 (depth < 60 for 30-bit keys,
// < 93 for 63-bit), rounded up to whole warps.
constexpr int level_seg(int key_bits) { return key_bits == 63 ? 192 : 128; }
// Segments a later CTA takes.
constexpr int level_fan(int key_bits) { return (kLevelItems - 1) / level_seg(key_bits); }

// Launches of later levels above `groups` groups.
constexpr int later_levels(int groups, int fan) {
  int lv = 0;
  for (; groups > 1; ++lv) groups = (groups + fan - 1) / fan;
  return lv;
}

// Leaves per CTA at the first level: the fewest that need no more levels than
// groups of 1,024 do.  A first level lasts as long as its CTAs' climbs, which
// grow with the group, and a later level about 10 us whatever it holds.  Both
// levels together: 36 us against 46 at n = 20,011 (256 leaves), 46 / 48 at 100,000
// (512), 110 / 119 at 1M (512).
constexpr int leaf_group(int n, int fan) {
  const int lv = later_levels((n + 1023) / 1024, fan);
  for (int g = 256; g < 1024; g *= 2)
    if (later_levels((n + g - 1) / g, fan) <= lv) return g;
  return 1024;
}

// First-level CTAs at most, for any n <= cap.  With fan^lv groups of 256 the
// lv later levels are full: more leaves take larger groups, as many at most,
// until the next level is worth it.
constexpr size_t max_groups(int cap, int fan) {
  const int g = leaf_group(cap, fan);
  size_t most = ((size_t)cap + g - 1) / g;
  for (size_t full = 1; 256 * full <= (size_t)cap; full *= fan)
    if (most < full) most = full;
  return most;
}
// For a workspace of `key_bits`; one of 63 bits also builds 30-bit trees.
constexpr size_t build_groups(int cap, int key_bits) {
  const size_t a = max_groups(cap, level_fan(30));
  const size_t b = key_bits == 63 ? max_groups(cap, level_fan(63)) : 0;
  return a > b ? a : b;
}
constexpr size_t build_seg_entries(int cap, int key_bits) {
  const size_t a = max_groups(cap, level_fan(30)) * level_seg(30);
  const size_t b = key_bits == 63 ? max_groups(cap, level_fan(63)) * level_seg(63) : 0;
  return a > b ? a : b;
}

}  // namespace nb
