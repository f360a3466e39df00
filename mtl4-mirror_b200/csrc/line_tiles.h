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

// Whether a factor's records may take `padded` bytes where its rows' own take
// `own`.  Lanes without a line and stages without a row are stored too: a plane of
// two lines takes 16 times its rows, lines of 8 rows 4 to 6 times.  Grids of ordinary
// shape stay below twice their rows.  Thin ones keep their records while these are a
// small part of the device's memory (a level-ordered sweep of such a grid has as
// many levels as the grid is long, and takes 1.3 us for each); beyond that their
// sweeps go by levels, at a few dozen bytes per row.
inline bool line_records_fit(long long own, long long padded, long long device) {
  return padded <= 4 * own || padded <= device / 32;
}

}  // namespace mtlgpu
