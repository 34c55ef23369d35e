"""A transform launch's set of fields refuses a field too many, and a launch
that takes one kind of field refuses a set of two kinds."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "web-exoplasim_b200", "csrc")

PROGRAM = r"""
#include "transform_set.h"
#include <cstdio>
#include <vector>
using namespace exogcm;
static bool refused(const std::vector<int>& opts) {
  try {
    TrSet s;
    for (int o : opts) {
      TrField t;
      t.planes = 3;
      t.opt = o;
      s.add(t);
    }
    const bool all = tr_every(s, [](const TrField& t) { return (t.opt & kTrDerivative) != 0; });
    if (all != (!opts.empty() && (opts[0] & kTrDerivative))) std::printf("wrong kind\n");
    if (tr_tiles(s, 2) != 2 * s.n) std::printf("wrong tiles\n");
  } catch (const std::logic_error&) { return true; }
  return false;
}
int main() {
  std::printf("%d %d %d %d %d %d %d\n", refused({}), refused(std::vector<int>(kMaxTr, 0)),
              refused(std::vector<int>(kMaxTr, 1)), refused(std::vector<int>(kMaxTr + 1, 0)), refused({0, 1}),
              refused({1, 1, 0}), refused({1, 1 | kTrKeep}));
}
"""


def test_sets_are_bounded_and_of_one_kind(tmp_path):
    source, program = tmp_path / "set.cpp", tmp_path / "set"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split() == \
        ["0", "0", "0", "1", "1", "1", "0"]
