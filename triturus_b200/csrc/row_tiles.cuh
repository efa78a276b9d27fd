// How the rows of a result are cut into tiles of whole units of 32 rows; plain C++, so that it can be checked without a GPU.
#pragma once

#ifdef __CUDACC__
#define TB200_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TB200_HOST_DEVICE inline
#endif

namespace tb200 {

// Tile `t` of `tiles` even ones over `units` units: the first `units % tiles` have one unit more.  (No product of the two:
// tile * units / tiles leaves 32 bits from 3.6 million rows on.)
struct RowTile {
  int first, units;
};
TB200_HOST_DEVICE RowTile row_tile(int units, int tiles, int t) {
  const int base = units / tiles, more = units - base * tiles;
  return {t * base + (t < more ? t : more), base + (t < more ? 1 : 0)};
}

}  // namespace tb200
