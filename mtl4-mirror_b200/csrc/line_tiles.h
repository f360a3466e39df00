// Which tiles of lines a grid-line sweep has (line_sweep.cu), as plain integer
// arithmetic for the host, the kernels and a test without a GPU.
//
// Line j of plane i stands at place js = j + i sk of its plane (sk: lines shifted
// per plane), so the grid is a sheared band: plane i covers i sk <= js < i sk + P.
// Tile row ti is the planes [ti TI, ti TI + TI); its tiles, TJ places wide and at
// multiples of TJ, are numbered from the first one the band meets.  A tile row's
// number of tiles therefore follows from P, not from the shear of the whole grid:
// a grid of 2,000 planes of 8 lines has 1,500 tiles, its sheared bounding box
// 125,500.
//
// Tiles are taken in ascending number.  A line depends on lines at the same or a
// lower js of the same or the previous plane, so on tiles of a lower number.
#pragma once

#include <numeric>

#ifdef __CUDACC__
#define MTLGPU_HD __host__ __device__ __forceinline__
#else
#define MTLGPU_HD inline
#endif

namespace mtlgpu {

// The column (js / TJ) of tile row ti's first tile.
MTLGPU_HD int line_tile_col0(int ti, int TI, int TJ, int sk) { return ti * TI * sk / TJ; }

// Tiles per tile row: the widest row's, whose band starts TJ - gcd(TI, TJ) places
// into its first tile.
inline int line_tile_cols(int P, int NI, int TI, int TJ, int sk) {
  const int planes = TI < NI ? TI : NI;
  return (sk * (TJ - std::gcd(TI, TJ)) + (planes - 1) * sk + P - 1) / TJ + 1;
}

inline long long line_tile_count(int P, int NI, int TI, int TJ, int sk) {
  return ((long long)NI + TI - 1) / TI * line_tile_cols(P, NI, TI, TJ, sk);
}

// The tile of line (i, js).
MTLGPU_HD long long line_tile_of(int i, int js, int TI, int TJ, int sk, int cols) {
  const int ti = i / TI;
  return (long long)ti * cols + js / TJ - line_tile_col0(ti, TI, TJ, sk);
}

}  // namespace mtlgpu
