"""When a handle captures its longer step graph (sdg_internal.h): not in calls of
a few dozen steps whose dt is new each time, but in a run of such calls that keep
their dt."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "scale-dg-kernel-extraction_b200", "csrc")

PROGRAM = r"""
#include <cassert>
#include "sdg_internal.h"

// Captures in `calls` calls of n steps: one dt, or a new one each call.
int captures(int calls, int n, bool new_dt) {
  int made = 0;
  bool have = false;
  long long asked = 0;
  for (int c = 0; c < calls; ++c) {
    if (new_dt) { have = false; asked = 0; }
    asked += n;
    if (!have && sdg::step_graph_pays(asked, n)) { have = true; ++made; }
  }
  return made;
}

int main() {
  for (int n : {1, 7, 8, 24, 32, 64, 100}) assert(captures(50, n, true) == 0);
  for (int n : {8, 24, 100, 128, 1000}) assert(captures(50, n, false) == 1);
  assert(captures(50, 7, false) == 0);     // never long enough to use it
  assert(captures(1, 128, true) == 1);
}
"""


def test_rule(tmp_path):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-I", CSRC, "-o", exe, src], check=True)
    subprocess.run([exe], check=True)
