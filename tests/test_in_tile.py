"""node_in_tile (sdg_in_tile.h) under the undefined-behaviour sanitiser: the
kernels' test for a face neighbour in the tile, at the limits of the node count
too, where the difference to a halo entry does not fit an int."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "scale-dg-kernel-extraction_b200", "csrc")

PROGRAM = r"""
#include <cassert>
#include <climits>
#include <initializer_list>
#include "sdg_in_tile.h"

int main() {
  using sdg::node_in_tile;
  const int np[] = {8, 512, 4096};
  for (int p : np) {
    const int last = INT_MAX / p - 1;  // element whose nodes still fit
    for (int e0 : {0, 7, last - 3}) {
      assert(node_in_tile(-1, e0, 3, p) == -1 && node_in_tile(INT_MIN + 1, e0, 3, p) == -1);
      assert(node_in_tile(INT_MIN, e0, 3, p) == -1);
      for (int s = 0; s < 3; ++s) assert(node_in_tile((e0 + s) * p, e0, 3, p) == s * p);
      assert(node_in_tile((e0 + 3) * p, e0, 3, p) == -1);
      if (e0 > 0) assert(node_in_tile((e0 - 1) * p, e0, 3, p) == -1);
      assert(node_in_tile(last * p, 0, 3, p) == -1 && node_in_tile(0, last - 3, 3, p) == -1);
    }
  }
}
"""


def test_limits(tmp_path):
    src, exe = tmp_path / "tile.cpp", tmp_path / "tile"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-fsanitize=undefined",
                    "-fno-sanitize-recover=all", "-I", CSRC, "-o", exe, src], check=True)
    subprocess.run([exe], check=True)


def test_kernels_use_it():
    for name in ("sdg_tend_line.cuh", "sdg_tend_warp32.cuh"):
        text = open(os.path.join(CSRC, name)).read()
        assert "node_in_tile(" in text, name
        assert not re.search(r"\bp[bf]? - \w+\.e0 \* NP", text), name
