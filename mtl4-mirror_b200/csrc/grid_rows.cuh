// Rows of a stencil matrix in a kernel (Sell's grid layout, sell.cu): the whole
// matrix has W distinct offsets (column - row), row r's entry at offset off[k]
// is val[((r / 128) W + k) 128 + r % 128], and bit k of the row's mask says
// whether it has one (no value is stored there otherwise).
//
// A thread takes a row.  The offsets are kernel parameters and a row's mask is 1,
// 2 or 4 bytes, so nothing a row needs is behind another load: its mask, its
// values and the vector elements are all issued at once.  A thread per row with
// an index per entry (spmv_sell and the SELL-32 forms of the other kernels)
// waits for the slice's place, then the indices, then the vector elements, and
// reads 2-4 more bytes per entry.  B200, before and after, us: FP64 product 128^3
// 7-point 28.3 / 22.5, 96^3 27-point 42.6 / 32.9, FP32 22.7 / 16.4 and 32.5 /
// 24.5; CG's direction product FP32 30.3 / 26.7 and 40.9 / 29.0.  Tried and
// slower: the offsets per slice, read by shuffle (spmv_sell's thread per row;
// 24-55 for the FP64 product by occupancy: ~245 instructions per warp and
// slice), four or two consecutive rows per thread with 16-byte loads (28.7-49),
// the next row's values loaded a turn ahead (no change to the direction product
// at 4 blocks per SM, 30.6 at 3).
//
// Entries are taken in ascending offset, the stored column order, and an
// absent one is skipped, not multiplied by zero: row sums keep the reference's
// bits (mat_vec_mult.hpp:666-688).
#pragma once

#include "device.cuh"
#include "internal.h"

namespace mtlgpu {

constexpr int kGridSlice = 128;   // rows per slice
constexpr int kGridOffsets = 32;  // most offsets

struct GridView {
  int n, W, mask_bytes;
  const uint8_t* mask;
  int off[kGridOffsets];
};

inline GridView grid_view(const Sell& S) {
  GridView v{};
  v.n = S.n;
  v.W = S.W;
  v.mask_bytes = S.mask_bytes;
  v.mask = S.d_mask;
  for (int k = 0; k < S.W; k++) v.off[k] = S.off[k];
  return v;
}

namespace dev {

// One row; W its matrix's offsets, known when compiled (0: any number).
template <typename T, int W>
struct GridRow {
  const GridView& A;
  int row;
  bool inner;           // every element the warp's rows reach exists (warp-uniform)
  unsigned mask;
  long long at;         // of the row's first value

  __device__ __forceinline__ GridRow(const GridView& a, int r) : A(a), row(r) {
    const int w0 = r - (int)(threadIdx.x & 31);
    const int last = A.off[(W ? W : A.W) - 1];
    inner = w0 + A.off[0] >= 0 && w0 + 31 < A.n && w0 + 31 + last < A.n;
    mask = 0;
    if (row < A.n) {
      if (A.mask_bytes == 1) mask = __ldg(A.mask + row);
      else if (A.mask_bytes == 2) mask = __ldg(reinterpret_cast<const uint16_t*>(A.mask) + row);
      else mask = __ldg(reinterpret_cast<const uint32_t*>(A.mask) + row);
    }
    at = (long long)(row / kGridSlice) * (W ? W : A.W) * kGridSlice + row % kGridSlice;
  }
  // Entries k0 to k0 + C - 1 of an inner row, for W = 0.  Chunks of 8 and what is
  // left in one of its own length: with the last offset repeated up to 8 (a
  // tridiagonal matrix issued 16 loads per row for 6) these matrices were slower
  // than on SELL-32; with a predicate per load the FP64 kernels spilled.  n = 2M, us,
  // SELL-32 / repeated / now: 3 offsets FP64 product 22.0 / 24.6 / 18.5, FP32 17.4 / 25.4 /
  // 14.9, FP32 apply 25.9 / 41.1 / 25.3, a mixed CG iteration 66 / 92 / 57; 6: FP64 23.1 /
  // 26.7 / 24.6, FP32 20.5 / 26.0 / 18.4; 11: 40.5 / 41.2 / 38.9, 35.0 / 39.9 / 24.6, 41.0 /
  // 44.9 / 32.1, 110 / 110 / 77; 19: 67.1 / 61.2 / 59.4, 51.2 / 55.3 / 35.2, 68.4 / 65.9 / 42.3,
  // 165 / 160 / 111; 31: 104.5 / 87.9 / 86.0, 77.9 / 71.4 / 53.2, 86.3 / 69.8 / 61.0, 228 / 176 / 147.
  template <int C, typename Get, typename Fold>
  __device__ __forceinline__ void part(const T* __restrict__ vp, int k0, Get get, Fold fold) const {
    T a[C];
    decltype(get(0)) g[C];
#pragma unroll
    for (int u = 0; u < C; u++) {
      a[u] = __ldlu(vp + (k0 + u) * kGridSlice);
      g[u] = get(row + A.off[k0 + u]);
    }
#pragma unroll
    for (int u = 0; u < C; u++)
      if (mask >> (k0 + u) & 1u) fold(a[u], g[u]);
  }
  // fold(a, g) over the row's entries in ascending offset, g = get(c) at the
  // entry's column c; C entries' loads are issued before the first is used.
  template <int C, typename Get, typename Fold>
  __device__ __forceinline__ void entries(const T* __restrict__ val, Get get, Fold fold) const {
    const T* vp = val + at;
    if (inner) {
      if (W) {
#pragma unroll
        for (int k0 = 0; k0 < W; k0 += C) {
          T a[C];
          decltype(get(0)) g[C];
#pragma unroll
          for (int u = 0; u < C; u++)
            if (k0 + u < W) {
              a[u] = __ldlu(vp + (k0 + u) * kGridSlice);
              g[u] = get(row + A.off[k0 + u]);
            }
#pragma unroll
          for (int u = 0; u < C; u++)
            if (k0 + u < W && (mask >> (k0 + u) & 1u)) fold(a[u], g[u]);
        }
      } else {
        static_assert(W || C == 8, "a remainder of 1 to 7");
        int k0 = 0;
        for (; k0 + C <= A.W; k0 += C) part<C>(vp, k0, get, fold);
        switch (A.W - k0) {  // the same for every thread
          case 1: part<1>(vp, k0, get, fold); break;
          case 2: part<2>(vp, k0, get, fold); break;
          case 3: part<3>(vp, k0, get, fold); break;
          case 4: part<4>(vp, k0, get, fold); break;
          case 5: part<5>(vp, k0, get, fold); break;
          case 6: part<6>(vp, k0, get, fold); break;
          case 7: part<7>(vp, k0, get, fold); break;
        }
      }
    } else {
      for (int k = 0; k < (W ? W : A.W); k++)
        if (mask >> k & 1u) fold(__ldlu(vp + k * kGridSlice), get(row + A.off[k]));
    }
  }
};

}  // namespace dev

// Blocks for a grid-stride loop of a thread per row: resident ones only
// (`per_sm` of them), as few as take the same number of turns.
inline int grid_blocks(Ctx* ctx, int n, int block, int per_sm) {
  const long long need = ((long long)n + block - 1) / block;
  const long long most = (long long)ctx->num_sms * per_sm;
  const long long turns = (need + most - 1) / most;
  return (int)(need < 1 ? 1 : (need + turns - 1) / turns);
}

// Launches by the number of offsets: those of 2-D and 3-D stencils' matrices and
// triangles, any other with W = 0.
#define MTLGPU_BY_MATRIX(COUNT, LAUNCH) \
  switch (COUNT) {                      \
    case 5: LAUNCH(5); break;           \
    case 7: LAUNCH(7); break;           \
    case 9: LAUNCH(9); break;           \
    case 27: LAUNCH(27); break;         \
    default: LAUNCH(0); break;          \
  }
#define MTLGPU_BY_TRIANGLE(COUNT, LAUNCH) \
  switch (COUNT) {                        \
    case 2: LAUNCH(2); break;             \
    case 3: LAUNCH(3); break;             \
    case 4: LAUNCH(4); break;             \
    case 13: LAUNCH(13); break;           \
    default: LAUNCH(0); break;            \
  }
constexpr int grid_chunk(int W) { return W == 27 ? 9 : W == 13 ? 7 : W ? W : 8; }

}  // namespace mtlgpu
