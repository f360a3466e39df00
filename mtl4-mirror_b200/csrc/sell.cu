// SELL-32: a sliced-ELL copy of a CSR matrix (or of a factor's off-diagonal
// part) for the streaming kernels of sm_100a.
//
// Rows are cut into slices of 32 consecutive rows; slice s stores
// width_s = (longest row of the slice) columns of entries column-major:
// entry k of row r sits at slice_ptr[s] + 32 k + (r mod 32).  Shorter rows
// are padded with column -1 (skipped by every kernel, so a padded slot never
// enters an arithmetic operation).  A warp owns a slice: its k-th load of
// column indices / values is one coalesced 128 / 256-byte line, and for
// stencil matrices the k-th gathers of x of 32 consecutive rows share the same
// offset, so they coalesce too.  Entries keep their CSR order inside each row,
// so a row processed in k order is processed in the reference's order.
//
// Grid layout (grid_rows.cuh).  A matrix with at most 32 distinct offsets
// (column - row), as a stencil has on a grid, needs no index per entry: its
// offsets are kept once, a row's mask says which it has, and the values go by
// offset in slices of 128 rows.  Chosen where storing every offset for every
// row takes at most kGridPadding times the stored entries; the values are then
// that much more, and the 2-4 bytes of index per entry are gone.
//
// Used by the SpMV (spmv.cu, for matrices whose padding is small) and by the
// Jacobi-iteration triangular solves (jacobi_sweep.cu, off-diagonal part with
// the diagonal kept apart).
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "device.cuh"
#include "grid_rows.cuh"
#include "internal.h"

namespace mtlgpu {

using namespace dev;

namespace {

constexpr int kBlock = 256;
constexpr double kGridPadding = 1.25;

int grid_rows(Ctx* ctx, long long n) {
  long long need = (n + kBlock - 1) / kBlock;
  long long cap = (long long)ctx->num_sms * 8;
  return (int)std::max(1ll, std::min(need, cap));
}

// diag_pos: 0 = no stored diagonal (unit lower), 1 = first entry of the row,
// 2 = last entry of the row.
__device__ __forceinline__ void off_range(const int32_t* rp, int r, int diag_pos, int& b, int& e) {
  b = rp[r];
  e = rp[r + 1];
  if (diag_pos == 1 && e > b) b++;
  if (diag_pos == 2 && e > b) e--;
}

// Slice widths (in entries per row) -> width32[s] = 32 * width.
__global__ void slice_width_kernel(int n, int n_slices, const int32_t* __restrict__ rp,
                                   int diag_pos, int32_t* __restrict__ width32) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = gtid() >> 5, nwarps = gstride() >> 5;
  for (long long s = warp0; s < n_slices; s += nwarps) {
    const long long r = s * 32 + lane;
    int cnt = 0;
    if (r < n) {
      int b, e;
      off_range(rp, (int)r, diag_pos, b, e);
      cnt = e - b;
    }
    for (int off = 16; off > 0; off >>= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, off));
    if (lane == 0) width32[s] = 32 * cnt;
  }
}

// The stored diagonal of row r (diag_pos 1: first entry, 2: last entry).
__device__ __forceinline__ double diag_of(const int32_t* rp, const double* v, int r,
                                          int diag_pos) {
  return v[diag_pos == 1 ? rp[r] : rp[r + 1] - 1];
}

// Scatter the off-diagonal entries into the slices; pad; copy the diagonal.
// scale_cols: each entry (r, c) is stored multiplied by the stored diagonal
// of row c (the factor N D of the Jacobi solves); with round64 both factors
// are the float values, whose product a double holds exactly.
__global__ void slice_fill_kernel(int n, const int32_t* __restrict__ rp,
                                  const int32_t* __restrict__ ci, const double* __restrict__ v,
                                  int diag_pos, const int32_t* __restrict__ slice_ptr,
                                  int32_t* __restrict__ col, double* __restrict__ val,
                                  float* __restrict__ val32, double* __restrict__ dinv,
                                  float* __restrict__ dinv32, bool round64, bool scale_cols) {
  for (long long r = gtid(); r < n; r += gstride()) {
    const long long s = r >> 5;
    const int lane = (int)(r & 31);
    const int base = slice_ptr[s], width = (slice_ptr[s + 1] - base) >> 5;
    int b, e;
    off_range(rp, (int)r, diag_pos, b, e);
    for (int k = 0; k < width; k++) {
      const int j = b + k;
      const long long o = base + 32ll * k + lane;
      const bool real = j < e;
      col[o] = real ? ci[j] : -1;
      double a = real ? v[j] : 0.0;
      // round64: the double copy holds the float values (FP32 factors are
      // applied at their float values, as the exact sweeps do)
      if (round64) a = (double)(float)a;
      if (scale_cols && real) {
        double dc = diag_of(rp, v, ci[j], diag_pos);
        if (round64) dc = (double)(float)dc;
        a *= dc;
      }
      if (val) val[o] = a;
      if (val32) val32[o] = (float)a;
    }
    if (diag_pos) {
      const double d = diag_of(rp, v, (int)r, diag_pos);
      if (dinv) dinv[r] = round64 ? (double)(float)d : d;
      if (dinv32) dinv32[r] = (float)d;
    }
  }
}

// The distinct offsets of a sample of rows: 128 runs of 32 consecutive rows,
// spread without a pattern that a grid's lines could share.  One block, so that
// the table (offset ^ 2^31, 0 = free) lives in shared memory: inserting every
// entry's offset from the whole grid took milliseconds of contended atomics.
// out: their number (kGridOffsets + 1: more), then the offsets.
constexpr int kSampleThreads = 1024, kSampleRuns = 4;
__global__ void __launch_bounds__(kSampleThreads)
    offsets_sample_kernel(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                          int diag_pos, int* __restrict__ out) {
  __shared__ unsigned table[kGridOffsets];
  __shared__ int over;
  if (threadIdx.x < kGridOffsets) table[threadIdx.x] = 0;
  if (threadIdx.x == 0) over = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = 0; q < kSampleRuns; q++) {
    const unsigned run = warp * kSampleRuns + q;
    const unsigned start = (unsigned)(((unsigned long long)(run * 2654435761u) * (unsigned)n) >> 32);
    const long long r = (long long)start + lane;
    if (r >= n) continue;
    int b, e;
    off_range(rp, (int)r, diag_pos, b, e);
    for (int j = b; j < e; j++) {
      if (((volatile int*)&over)[0]) break;
      const unsigned d = (unsigned)(ci[j] - (int)r) ^ 0x80000000u;
      int k = 0;
      for (; k < kGridOffsets; k++) {
        unsigned t = ((volatile unsigned*)table)[k];
        if (t == 0) t = atomicCAS(table + k, 0u, d);
        if (t == 0 || t == d) break;
      }
      if (k == kGridOffsets) over = 1;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int cnt = 0;
    for (int k = 0; k < kGridOffsets && table[k]; k++) out[1 + cnt++] = (int)(table[k] ^ 0x80000000u);
    out[0] = over ? kGridOffsets + 1 : cnt;
  }
}

// *missing is set when an entry lies at none of G's offsets or a row is not
// sorted; *count gets the entries.
__global__ void offsets_verify_kernel(GridView G, const int32_t* __restrict__ rp,
                                      const int32_t* __restrict__ ci, int diag_pos,
                                      unsigned long long* count, int* missing) {
  unsigned long long cnt = 0;
  for (long long r = gtid(); r < G.n; r += gstride()) {
    if (ld_relaxed(missing)) break;
    int b, e;
    off_range(rp, (int)r, diag_pos, b, e);
    cnt += e - b;
    int k = 0;
    for (; b < e; b++) {
      const int d = ci[b] - (int)r;
      while (k < G.W && G.off[k] != d) k++;
      if (k++ >= G.W) {
        st_relaxed(missing, 1);
        break;
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(count, cnt);
}

// Masks (when given), values and diagonals of the grid layout.
__global__ void grid_fill_kernel(GridView G, const int32_t* __restrict__ rp,
                                 const int32_t* __restrict__ ci, const double* __restrict__ v,
                                 int diag_pos, uint8_t* __restrict__ mask,
                                 double* __restrict__ val, float* __restrict__ val32,
                                 double* __restrict__ dinv, float* __restrict__ dinv32,
                                 bool round64, bool scale_cols) {
  for (long long r = gtid(); r < G.n; r += gstride()) {
    int b, e;
    off_range(rp, (int)r, diag_pos, b, e);
    unsigned m = 0;
    const long long o = r / kGridSlice * G.W * kGridSlice + r % kGridSlice;
    for (int k = 0; k < G.W; k++) {
      double a = 0.0;
      if (b < e && ci[b] - (int)r == G.off[k]) {
        m |= 1u << k;
        a = v[b];
        // round64: the double copy holds the float values (slice_fill_kernel)
        if (round64) a = (double)(float)a;
        if (scale_cols) {
          double dc = diag_of(rp, v, ci[b], diag_pos);
          if (round64) dc = (double)(float)dc;
          a *= dc;
        }
        b++;
      }
      if (val) val[o + (long long)k * kGridSlice] = a;
      if (val32) val32[o + (long long)k * kGridSlice] = (float)a;
    }
    if (mask) {
      if (G.mask_bytes == 1) mask[r] = (uint8_t)m;
      if (G.mask_bytes == 2) reinterpret_cast<uint16_t*>(mask)[r] = (uint16_t)m;
      if (G.mask_bytes == 4) reinterpret_cast<uint32_t*>(mask)[r] = m;
    }
    if (diag_pos) {
      const double d = diag_of(rp, v, (int)r, diag_pos);
      if (dinv) dinv[r] = round64 ? (double)(float)d : d;
      if (dinv32) dinv32[r] = (float)d;
    }
  }
}

// Largest |column - row| over the stored entries (padding skipped).
__global__ void delta_max_kernel(int n, const int32_t* __restrict__ slice_ptr,
                                 const int32_t* __restrict__ col, int* __restrict__ out) {
  int m = 0;
  for (long long r = gtid(); r < n; r += gstride()) {
    const long long s = r >> 5;
    const int lane = (int)(r & 31);
    const int base = slice_ptr[s], width = (slice_ptr[s + 1] - base) >> 5;
    for (int k = 0; k < width; k++) {
      const int c = col[base + 32 * k + lane];
      if (c >= 0) m = max(m, abs(c - (int)r));
    }
  }
  for (int off = 16; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// 16-bit column deltas: column - row, padding -32768.
__global__ void dcol_fill_kernel(int n, const int32_t* __restrict__ slice_ptr,
                                 const int32_t* __restrict__ col, int16_t* __restrict__ dcol) {
  for (long long r = gtid(); r < n; r += gstride()) {
    const long long s = r >> 5;
    const int lane = (int)(r & 31);
    const int base = slice_ptr[s], width = (slice_ptr[s + 1] - base) >> 5;
    for (int k = 0; k < width; k++) {
      const int o = base + 32 * k + lane;
      const int c = col[o];
      dcol[o] = (int16_t)(c >= 0 ? c - (int)r : -32768);
    }
  }
}

}  // namespace

// MTLGPU_SELL_INDEX=32 keeps a 32-bit index per entry.
static bool wide_indices_asked() {
  const char* m = std::getenv("MTLGPU_SELL_INDEX");
  return m && std::atoi(m) == 32;
}

static mtlgpu_status grid_fill(Ctx* ctx, const int32_t* d_rp, const int32_t* d_ci,
                               const double* d_v, int diag_pos, Sell* J, bool masks) {
  grid_fill_kernel<<<grid_rows(ctx, J->n), kBlock, 0, ctx->stream>>>(
      grid_view(*J), d_rp, d_ci, d_v, diag_pos, masks ? J->d_mask : nullptr, J->d_val, J->d_val32,
      J->d_dinv, J->d_dinv32, J->round64, J->col_scaled);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return MTLGPU_OK;
}

// The distinct offsets (column - row) of a sample of the rows, ascending; *count
// is kGridOffsets + 1 when there are more.  Who uses them looks at every row.
mtlgpu_status sample_offsets(Ctx* ctx, int n, const int32_t* d_rp, const int32_t* d_ci,
                             int diag_pos, int* off, int* count) {
  int h[kGridOffsets + 1], *d = nullptr;
  MTLGPU_TRY(dalloc(ctx, &d, kGridOffsets + 1));
  offsets_sample_kernel<<<1, kSampleThreads, 0, ctx->stream>>>(n, d_rp, d_ci, diag_pos, d);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  dfree(ctx, d);
  *count = h[0];
  if (h[0] <= kGridOffsets) {
    std::copy(h + 1, h + 1 + h[0], off);
    std::sort(off, off + h[0]);
  }
  return MTLGPU_OK;
}

// Takes the grid layout when the pattern has few enough offsets and little
// enough padding; J->grid says whether it did.
static mtlgpu_status grid_build(Ctx* ctx, const int32_t* d_rp, const int32_t* d_ci,
                                const double* d_v, int diag_pos, bool fp64, bool fp32, Sell* J) {
  if (wide_indices_asked()) return MTLGPU_OK;
  int off[kGridOffsets], W = 0;
  MTLGPU_TRY(sample_offsets(ctx, J->n, d_rp, d_ci, diag_pos, off, &W));
  if (W == 0 || W > kGridOffsets) return MTLGPU_OK;
  J->W = W;
  std::copy(off, off + W, J->off);
  struct {
    unsigned long long count;
    int missing, pad;
  } h, *d = nullptr;
  MTLGPU_TRY(dalloc(ctx, &d, 1));
  MTLGPU_TRY_CUDA(ctx, cudaMemsetAsync(d, 0, sizeof(h), ctx->stream));
  offsets_verify_kernel<<<grid_rows(ctx, J->n), kBlock, 0, ctx->stream>>>(
      grid_view(*J), d_rp, d_ci, diag_pos, &d->count, &d->missing);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  dfree(ctx, d);
  const long long slices = ((long long)J->n + kGridSlice - 1) / kGridSlice;
  if (h.missing || (double)W * J->n > kGridPadding * (double)h.count) {
    J->W = 0;
    return MTLGPU_OK;
  }
  J->grid = true;
  J->max_width = W;
  J->mask_bytes = W <= 8 ? 1 : W <= 16 ? 2 : 4;
  J->n_ent = slices * kGridSlice * W;
  const size_t rows = (size_t)slices * kGridSlice;
  MTLGPU_TRY(dalloc(ctx, &J->d_mask, rows * J->mask_bytes));
  if (rows > (size_t)J->n)  // rows past the end have no entries
    MTLGPU_TRY_CUDA(ctx, cudaMemsetAsync(J->d_mask + (size_t)J->n * J->mask_bytes, 0,
                                         (rows - J->n) * J->mask_bytes, ctx->stream));
  if (fp64) MTLGPU_TRY(dalloc(ctx, &J->d_val, J->n_ent));
  if (fp32) MTLGPU_TRY(dalloc(ctx, &J->d_val32, J->n_ent));
  if (diag_pos) {
    if (fp64) MTLGPU_TRY(dalloc(ctx, &J->d_dinv, J->n));
    if (fp32) MTLGPU_TRY(dalloc(ctx, &J->d_dinv32, J->n));
  }
  return grid_fill(ctx, d_rp, d_ci, d_v, diag_pos, J, true);
}

// Builds J->d_dcol when every stored entry lies within 32,767 of its row.
static mtlgpu_status sell_build_deltas(Ctx* ctx, Sell* J) {
  if (wide_indices_asked()) return MTLGPU_OK;
  int* d_max = nullptr;
  MTLGPU_TRY(dalloc(ctx, &d_max, 1));
  MTLGPU_TRY_CUDA(ctx, cudaMemsetAsync(d_max, 0, sizeof(int), ctx->stream));
  delta_max_kernel<<<grid_rows(ctx, J->n), kBlock, 0, ctx->stream>>>(J->n, J->d_slice_ptr,
                                                                      J->d_col, d_max);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  int h_max = 0;
  MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(&h_max, d_max, sizeof(int), cudaMemcpyDeviceToHost,
                                       ctx->stream));
  MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  dfree(ctx, d_max);
  if (h_max > 32767) return MTLGPU_OK;
  MTLGPU_TRY(dalloc(ctx, &J->d_dcol, J->n_ent));
  dcol_fill_kernel<<<grid_rows(ctx, J->n), kBlock, 0, ctx->stream>>>(J->n, J->d_slice_ptr,
                                                                      J->d_col, J->d_dcol);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return MTLGPU_OK;
}

// Padded entry count of the SELL-32 form of a CSR pattern (diag_pos as
// sell_build), from host row pointers.
long long sell_padded_entries(int n, const int32_t* h_rp, int diag_pos) {
  long long total = 0;
  for (int s = 0; s * 32 < n; s++) {
    int w = 0;
    for (int r = s * 32; r < std::min(n, s * 32 + 32); r++) {
      int len = h_rp[r + 1] - h_rp[r];
      if (diag_pos && len > 0) len--;
      w = std::max(w, len);
    }
    total += 32ll * w;
  }
  return total;
}

// fp64 / fp32: which value copies to hold; round64: the double copy holds
// the float-rounded values (FP32 factors); scale_cols: entries stored times
// the stored diagonal of their column's row (needs diag_pos != 0).
mtlgpu_status sell_build(Ctx* ctx, int n, const int32_t* d_rp, const int32_t* d_ci,
                         const double* d_v, int diag_pos, bool fp64, bool fp32, bool round64,
                         bool scale_cols, bool grid_ok, Sell* J) {
  J->n = n;
  J->round64 = round64;
  J->col_scaled = scale_cols && diag_pos != 0;
  J->unit_diag = diag_pos == 0;
  J->n_slices = (n + 31) / 32;
  if (n == 0) return MTLGPU_OK;
  if (grid_ok) {
    MTLGPU_TRY(grid_build(ctx, d_rp, d_ci, d_v, diag_pos, fp64, fp32, J));
    if (J->grid) return MTLGPU_OK;
  }
  int32_t* d_w = nullptr;
  MTLGPU_TRY(dalloc(ctx, &d_w, J->n_slices + 1));
  MTLGPU_TRY_CUDA(ctx, cudaMemsetAsync(d_w, 0, sizeof(int32_t) * (J->n_slices + 1), ctx->stream));
  slice_width_kernel<<<grid_rows(ctx, 32ll * J->n_slices), kBlock, 0, ctx->stream>>>(
      n, J->n_slices, d_rp, diag_pos, d_w);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  MTLGPU_TRY(dalloc(ctx, &J->d_slice_ptr, J->n_slices + 1));
  MTLGPU_TRY(scan_i32(ctx, d_w, J->d_slice_ptr, J->n_slices + 1));
  {
    std::vector<int32_t> hw(J->n_slices);
    MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(hw.data(), d_w, sizeof(int32_t) * J->n_slices,
                                         cudaMemcpyDeviceToHost, ctx->stream));
    MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    int mx = 0;
    for (int32_t w : hw) mx = std::max(mx, (int)(w / 32));
    J->max_width = mx;
  }
  dfree(ctx, d_w);
  int total = 0;
  MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(&total, J->d_slice_ptr + J->n_slices, sizeof(int),
                                       cudaMemcpyDeviceToHost, ctx->stream));
  MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (total < 0) return MTLGPU_NOT_SUPPORTED;  // more than 2^31 padded entries
  J->n_ent = total;
  MTLGPU_TRY(dalloc(ctx, &J->d_col, total));
  if (fp64) MTLGPU_TRY(dalloc(ctx, &J->d_val, total));
  if (fp32) MTLGPU_TRY(dalloc(ctx, &J->d_val32, total));
  if (diag_pos) {
    if (fp64) MTLGPU_TRY(dalloc(ctx, &J->d_dinv, n));
    if (fp32) MTLGPU_TRY(dalloc(ctx, &J->d_dinv32, n));
  }
  slice_fill_kernel<<<grid_rows(ctx, n), kBlock, 0, ctx->stream>>>(
      n, d_rp, d_ci, d_v, diag_pos, J->d_slice_ptr, J->d_col, J->d_val, J->d_val32, J->d_dinv,
      J->d_dinv32, J->round64, J->col_scaled);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return sell_build_deltas(ctx, J);
}

void sell_free(Ctx* ctx, Sell* J) {
  dfree(ctx, J->d_slice_ptr);
  dfree(ctx, J->d_col);
  dfree(ctx, J->d_dcol);
  dfree(ctx, J->d_mask);
  dfree(ctx, J->d_val);
  dfree(ctx, J->d_val32);
  dfree(ctx, J->d_dinv);
  dfree(ctx, J->d_dinv32);
  *J = Sell();
}

// New values on the same pattern (mtlgpu_csr_set_values).
mtlgpu_status sell_refill(Ctx* ctx, const int32_t* d_rp, const int32_t* d_ci, const double* d_v,
                          int diag_pos, Sell* J) {
  if (J->n == 0) return MTLGPU_OK;
  if (J->grid) return grid_fill(ctx, d_rp, d_ci, d_v, diag_pos, J, false);
  slice_fill_kernel<<<grid_rows(ctx, J->n), kBlock, 0, ctx->stream>>>(
      J->n, d_rp, d_ci, d_v, diag_pos, J->d_slice_ptr, J->d_col, J->d_val, J->d_val32, J->d_dinv,
      J->d_dinv32, J->round64, J->col_scaled);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return MTLGPU_OK;
}

// Adds the float copy of the values (mixed-precision solves) when missing.
mtlgpu_status sell_ensure_fp32(Ctx* ctx, const int32_t* d_rp, const int32_t* d_ci,
                               const double* d_v, int diag_pos, Sell* J) {
  if (J->n == 0 || J->d_val32) return MTLGPU_OK;
  MTLGPU_TRY(dalloc(ctx, &J->d_val32, J->n_ent));
  if (diag_pos) MTLGPU_TRY(dalloc(ctx, &J->d_dinv32, J->n));
  return sell_refill(ctx, d_rp, d_ci, d_v, diag_pos, J);
}

}  // namespace mtlgpu
