"""Room for the tree build's open splits (csrc/build_geometry.h), host side only:
a workspace reserved for `cap` particles serves every tree of up to `cap`, at both
key widths, and holds little more than the worst of them needs."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include "build_geometry.h"
using namespace nb;
int main() {
  // running maxima over n of what a tree of n needs, against the bounds at cap = n
  size_t g30 = 0, g63 = 0, s30 = 0, s63 = 0, bad = 0, loose = 0;
  for (int n = 2; n <= 4300000; ++n) {
    for (int bits : {30, 63}) {
      const int g = leaf_group(n, level_fan(bits));
      const size_t groups = ((size_t)n + g - 1) / g;
      size_t& most = bits == 63 ? g63 : g30;
      most = std::max(most, groups);
    }
    s30 = g30 * level_seg(30);
    s63 = std::max(s30, g63 * level_seg(63));
    bad += build_groups(n, 30) < g30 || build_groups(n, 63) < std::max(g30, g63);
    bad += build_seg_entries(n, 30) < s30 || build_seg_entries(n, 63) < s63;
    loose += build_groups(n, 30) > g30 || build_seg_entries(n, 63) > s63;
  }
  std::printf("%zu %zu %zu %zu\n", bad, loose, build_groups(1000000, 30),
              build_seg_entries(1000000, 30));
}
"""


def test_room_for_every_smaller_tree(tmp_path):
    (tmp_path / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I",
                    os.path.join(ROOT, "nbodyssey_b200", "csrc"), str(tmp_path / "m.cpp"),
                    "-o", str(tmp_path / "m")], check=True)
    bad, loose, groups, entries = map(int, subprocess.run(
        [str(tmp_path / "m")], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and loose == 0
    # 15^3 groups of 256 leaves are the most that up to 1,000,000 particles take
    assert groups == 15 ** 3 and entries == groups * 128
