// Neighbours inside a tile, shared by the kernels that read them from shared
// memory; plain C++ as well, so that the host can check it.
#pragma once

#ifdef __CUDACC__
#define SDG_HD __host__ __device__ __forceinline__
#else
#define SDG_HD inline
#endif

namespace sdg {

// First node, counted from the first of a tile (n elements of np nodes from e0
// on), of the neighbour element whose pbase entry is pb; -1: a halo face (pb < 0)
// or an element outside the tile.  All nodes of a mesh are counted in an int, so
// the difference of two of them fits, that of a halo entry and a node may not.
SDG_HD int node_in_tile(int pb, int e0, int n, int np) {
  if (pb < 0) return -1;
  const int d = pb - e0 * np;
  return d >= 0 && d < n * np ? d : -1;
}

}  // namespace sdg
