// Tiles of the grid-line sweeps (csrc/line_tiles.h) by brute force: every line
// has a tile, no two tiles share a place, dependencies point to the same or an
// earlier tile, and the number of tiles follows the number of lines on grids of
// any shape, in 64 bits.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "line_tiles.h"

using namespace mtlgpu;

static void check(bool ok, const char* what, int P, int NI, int TI, int TJ, int sk) {
  if (ok) return;
  std::printf("%s: P %d NI %d TI %d TJ %d sk %d\n", what, P, NI, TI, TJ, sk);
  std::exit(1);
}

static void grid(int P, int NI, int TI, int TJ, int sk, bool lines) {
  const int cols = line_tile_cols(P, NI, TI, TJ, sk);
  const long long count = line_tile_count(P, NI, TI, TJ, sk);
  // the band of a tile row is P + TI - 1 places wide, and each end of it may lie
  // inside a tile
  const long long rows = ((long long)NI + TI - 1) / TI;
  check(count == rows * cols, "count", P, NI, TI, TJ, sk);
  check(cols <= (P + sk * (TI - 1) + 2 * (TJ - 1)) / TJ + 1, "too many tiles", P, NI, TI, TJ, sk);
  if (!lines) return;
  for (int i = 0; i < NI; i++)
    for (int j = 0; j < P; j++) {
      const int js = j + i * sk;
      const long long t = line_tile_of(i, js, TI, TJ, sk, cols);
      check(t >= 0 && t < count, "tile out of range", P, NI, TI, TJ, sk);
      // the kernel's place of this tile, from its number
      const int ti = (int)(t / cols), J0 = (line_tile_col0(ti, TI, TJ, sk) + (int)(t % cols)) * TJ;
      check(i >= ti * TI && i < ti * TI + TI && js >= J0 && js < J0 + TJ, "place", P, NI, TI, TJ, sk);
      for (int a = 0; a <= 1; a++)
        for (int b = -1; b <= 1; b++) {
          if (a == 0 && b < 1) continue;
          const int di = i - a, dj = j - b;
          if (di < 0 || dj < 0 || dj >= P || (sk == 0 && a && b)) continue;
          check(line_tile_of(di, dj + di * sk, TI, TJ, sk, cols) <= t, "order", P, NI, TI, TJ, sk);
        }
    }
}

int main() {
  const int TI[] = {1, 4, 8, 16};
  for (int sk = 0; sk <= 1; sk++)
    for (int ti : TI)
      for (int P = 1; P <= 40; P++)
        for (int NI : {1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 33, 100})
          grid(P, NI, ti, ti == 1 ? 32 : 8, sk, true);
  grid(8, 20000, 4, 8, 1, true);
  // sheared bounding boxes of more than 2^31 tiles
  grid(3, 262144, 4, 8, 1, false);
  grid(3, 370728, 4, 8, 1, false);
  grid(3, 80000000, 4, 8, 1, false);
  check(line_tile_count(3, 370728, 4, 8, 1) <= 2ll * 370728 / 4, "linear", 3, 370728, 4, 8, 1);
  // records: up to four times the rows' own, or a 32nd of the device
  const long long device = 180ll << 30, part = device / 32;
  for (long long own : {1ll << 20, part / 4 + 1, 40ll << 30})
    for (long long f : {1, 4, 5, 16}) {
      const bool fits = line_records_fit(own, f * own, device);
      if (fits != (f <= 4 || f * own <= part)) {
        std::printf("records %lld x %lld\n", own, f);
        return 1;
      }
    }
  std::puts("ok");
}
