"""The division of all-pairs scratch among simulations (csrc/scratch_share.h)."""
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "scratch_share.h"
// argv: total, then least and whole of each; prints the shares
int main(int argc, char** v) {
  std::vector<size_t> least, whole;
  for (int i = 2; i + 1 < argc; i += 2) {
    least.push_back(std::strtoull(v[i], nullptr, 10));
    whole.push_back(std::strtoull(v[i + 1], nullptr, 10));
  }
  for (size_t x : nb::share_scratch(least, whole, std::strtoull(v[1], nullptr, 10)))
    std::printf("%zu ", x);
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("share")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "nbodyssey_b200", "csrc"),
                    str(d / "m.cpp"), "-o", str(d / "m")], check=True)

    def run(total, pairs):
        args = [str(total)] + [str(x) for p in pairs for x in p]
        out = subprocess.run([str(d / "m")] + args, check=True, capture_output=True, text=True)
        return [int(x) for x in out.stdout.split()]
    return run


def test_shares_by_hand(share):
    assert share(100, []) == []
    assert share(100, [(3, 100)]) == [100]
    assert share(99, [(3, 100)]) == [99]
    assert share(100, [(3, 60), (2, 40)]) == [60, 40]
    assert share(55, [(5, 55), (0, 50), (10, 10)]) == [25, 20, 10]
    assert share(4, [(3, 60), (2, 40)]) == [3, 2]     # the caller's to refuse
    assert share(0, [(3, 60), (2, 40)]) == [3, 2]


def test_shares_of_any_pool(share):
    rng = random.Random(1)
    for _ in range(60):
        pairs = []
        for _ in range(rng.randint(1, 40)):
            low = rng.randint(0, 1 << rng.randint(0, 40))
            pairs.append((low, low + rng.randint(0, 1 << rng.randint(0, 50))))
        low, high = sum(p[0] for p in pairs), sum(p[1] for p in pairs)
        total = rng.randint(low, high + 10)
        got = share(total, pairs)
        assert all(a <= x <= b for x, (a, b) in zip(got, pairs))
        assert sum(got) <= total
        assert sum(got) > min(total, high) - len(pairs)   # rounded down, each by less than one
