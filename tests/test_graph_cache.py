"""Which batch shapes get a graph: the rule of csrc/graph_cache.h, run on the CPU."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "rust_trainer_b200" / "csrc"
HARNESS = r"""
#include <cstdlib>
#include <cstdio>
#include "graph_cache.h"
// shapes in argv order; what each pass does as the model does it: r(eplay), c(apture), e(ager)
int main(int argc, char** argv) {
  rt::GraphCache<int, int, 4> g;
  for (int i = 1; i < argc; ++i) {
    const int s = atoi(argv[i]);
    if (int* have = g.find(s)) {
      if (*have != s) return 1;
      putchar('r');
    } else if (g.worth_capturing(s)) {
      auto gone = g.put(s, s);
      if (gone && g.find(*gone)) return 2;
      putchar('c');
    } else {
      g.touch(s);
      putchar('e');
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def passes(tmp_path_factory):
    d = tmp_path_factory.mktemp("graphs")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "h.cpp"), "-o", str(d / "h")], check=True)
    return lambda shapes: subprocess.run([str(d / "h"), *map(str, shapes)], check=True, capture_output=True, text=True).stdout


@pytest.mark.parametrize("n", [1, 2, 4])
def test_shapes_that_fit_replay_from_the_third_time_on(passes, n):
    assert passes(list(range(n)) * 4) == "e" * n + "c" * n + "r" * (2 * n)


@pytest.mark.parametrize("n", [5, 7, 8, 64])
def test_a_cycle_of_more_shapes_than_places_is_not_captured_again_and_again(passes, n):
    assert passes(list(range(n)) * 5) == "e" * (5 * n)
    # shapes that had a graph before the cycle began keep it
    assert passes([0, 1, 2, 3] * 2 + list(range(n)) * 5) == "eeeecccc" + ("rrrr" + "e" * (n - 4)) * 5


def test_the_least_recently_used_graph_gives_way(passes):
    assert passes([0, 0, 1, 1, 2, 2, 3, 3, 0, 9, 9, 0, 2, 3, 9, 1]) == "ecececec" + "r" + "ec" + "rrrr" + "e"
