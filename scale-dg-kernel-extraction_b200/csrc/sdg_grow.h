// Growth of device tables that belong together.  The capacity counts only once
// every table of it is there: after a failed allocation it is 0, so that the
// next call allocates again instead of using what is missing or was freed.
#pragma once

#include <cstddef>

namespace sdg {

struct GrowTable {
  void** p;     // the table, null while there is none
  size_t each;  // bytes per unit of capacity
};

// Makes room for `need` units in the n tables (contents are not kept).
// alloc(void**, size_t) returns 0 or an error code, which this returns.
template <typename Alloc, typename Release>
int grow_tables(int need, int* cap, const GrowTable* t, int n, Alloc alloc, Release release) {
  if (need <= *cap) return 0;
  const int want = need > 2 * *cap ? need : 2 * *cap;
  *cap = 0;
  for (int i = 0; i < n; ++i) {
    if (*t[i].p) release(*t[i].p);
    *t[i].p = nullptr;
  }
  for (int i = 0; i < n; ++i)
    if (int rc = alloc(t[i].p, static_cast<size_t>(want) * t[i].each)) {
      *t[i].p = nullptr;
      return rc;
    }
  *cap = want;
  return 0;
}

}  // namespace sdg
