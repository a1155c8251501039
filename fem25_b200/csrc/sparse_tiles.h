// Tile geometry of the sparse factorisation's products (k_sp_gemm), the same on the
// device and on the host.
#pragma once

#ifdef __CUDACC__
#define FEM25_HD __host__ __device__ __forceinline__
#else
#define FEM25_HD inline
#endif

namespace fem25 {
namespace sp {

constexpr int kGt = 32;  // rows and columns of a product tile

// First row and column of tile `tile` of an M x M product whose launch covers the tile
// columns [c0, c0 + cn); entries with both indices >= corner are left alone (corner = M:
// none are).  False: the tile lies outside, or has nothing to do; M = 0 (a front
// without a boundary, after its last panel or in F22's product) has no tile at all.
FEM25_HD bool gemm_tile(int M, int corner, int tile, int c0, int cn, int *m0, int *n0) {
  if (M <= 0) return false;
  const int tiles = (M + kGt - 1) / kGt;
  const int tc = tile / tiles;
  if (tc >= cn || c0 + tc >= tiles) return false;
  *m0 = (tile - tc * tiles) * kGt;
  *n0 = (c0 + tc) * kGt;
  return *m0 < corner || *n0 < corner;
}

}  // namespace sp
}  // namespace fem25
