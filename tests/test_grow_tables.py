"""Growth of the batch's device tables (sdg_grow.h) with an allocator that
fails: the capacity must not count until every table is there, so that the next
call allocates them again."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "scale-dg-kernel-extraction_b200", "csrc")

PROGRAM = r"""
#include <cassert>
#include <cstdlib>
#include <set>
#include "sdg_grow.h"

int main() {
  std::set<void*> live;
  for (int fail_at = 0; fail_at < 2; ++fail_at) {
    void *insts = nullptr, *maps = nullptr;
    int cap = 0, calls = 0, failing = -1;
    auto alloc = [&](void** p, size_t bytes) {
      if (calls++ == failing) { *p = reinterpret_cast<void*>(16); return 2; }
      *p = std::malloc(bytes);
      live.insert(*p);
      return 0;
    };
    auto release = [&](void* p) { assert(live.erase(p) == 1); std::free(p); };
    const sdg::GrowTable t[2] = {{&insts, 24}, {&maps, 1536}};
    assert(sdg::grow_tables(3, &cap, t, 2, alloc, release) == 0 && cap == 3 && insts && maps);
    void* kept = maps;
    assert(sdg::grow_tables(2, &cap, t, 2, alloc, release) == 0 && maps == kept);
    calls = 0;
    failing = fail_at;  // the first or the second table does not come
    assert(sdg::grow_tables(4, &cap, t, 2, alloc, release) == 2);
    assert(cap == 0 && maps == nullptr && (fail_at == 1) == (insts != nullptr));
    failing = -1;       // memory is back, for no more than there was before
    assert(sdg::grow_tables(3, &cap, t, 2, alloc, release) == 0);
    assert(cap == 3 && insts && maps && live.size() == 2);
    release(insts);
    release(maps);
  }
}
"""


def test_capacity_counts_only_complete_tables(tmp_path):
    src, exe = tmp_path / "grow.cpp", tmp_path / "grow"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-I", CSRC, "-o", exe, src], check=True)
    subprocess.run([exe], check=True)
