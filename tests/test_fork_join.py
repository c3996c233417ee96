"""The two-stream step of a batch (csrc/fork_join.h), host control flow only:
whatever part fails, the first stream is ordered behind the second once the
second may hold work."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "fork_join.h"
// argv: has_side, then the statuses of fork, side, work, join, and whether
// work uses the second stream; prints the parts that ran and the result
int main(int, char** v) {
  auto part = [&](const char* name, int i) { std::printf("%s ", name); return std::atoi(v[i]); };
  const int rc = nb::run_forked(
      std::atoi(v[1]) != 0, [&] { return part("fork", 2); }, [&] { return part("side", 3); },
      [&](bool* used) { if (std::atoi(v[6])) *used = true; return part("work", 4); },
      [&] { return part("join", 5); });
  std::printf("%d\n", rc);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("fork")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "nbodyssey_b200", "csrc"),
                    str(d / "m.cpp"), "-o", str(d / "m")], check=True)
    return str(d / "m")


@pytest.mark.parametrize("has_side,fork,side,work,join,uses,ran", [
    (1, 0, 0, 0, 0, 0, "fork side work join 0"),
    (1, 0, 0, 0, 0, 1, "fork side work join 0"),
    (1, 0, 5, 0, 0, 0, "fork side join 5"),        # side failed with work queued before
    (1, 0, 5, 0, 6, 0, "fork side join 5"),
    (1, 4, 0, 0, 0, 0, "fork 4"),                  # never forked: nothing to join
    (1, 0, 0, 7, 0, 0, "fork side work join 7"),
    (1, 0, 0, 0, 6, 0, "fork side work join 6"),
    (0, 0, 0, 0, 0, 0, "work 0"),
    (0, 0, 0, 0, 0, 1, "work join 0"),
    (0, 0, 0, 7, 0, 1, "work join 7"),
    (0, 0, 0, 7, 0, 0, "work 7"),
])
def test_join_on_every_path(program, has_side, fork, side, work, join, uses, ran):
    args = [str(x) for x in (has_side, fork, side, work, join, uses)]
    out = subprocess.run([program] + args, check=True, capture_output=True, text=True).stdout
    assert out.strip() == ran
