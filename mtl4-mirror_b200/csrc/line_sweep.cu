// Triangular sweeps along grid lines for sm_100a.
//
// Same arithmetic as lower_trisolve_t::apply(int_<5>/<6>) and
// upper_trisolve_t::apply(int_<3>) (mtl/operation/lower_trisolve.hpp:173-209,
// upper_trisolve.hpp:160-176): for each row r in dependency order
//     rr = v[r];  for each off-diagonal entry j (stored order): rr -= F[r][j] * w[j];
//     w[r] = rr * dia[r]        (no multiply for a unit diagonal)
// with every multiply and subtract rounded separately: bit-identical to the
// reference's sequential loops, and to sweep.cu.
//
// For which factors.  Those of a stencil on a grid in natural order, found
// from the pattern alone: a line length B and a number P of lines per plane
// such that the entries of row r, apart from its predecessor's, lie on G other
// lines -- a planes and b lines back, a in {0,1}, b in {-1,0,1} -- at the same
// place (5- and 7-point) or at all three places next to it (9- and 27-point),
// and an entry is missing exactly where its place lies outside the grid
// (line_verify_kernel looks at every row).  The rows are taken in dependency order
// x = r for a lower factor, n-1-r for an upper one.
//
// Why.  The dependency chain of such a factor runs over B + P + N places (382
// levels on a 128^3 grid).  The level-ordered sweep (sweep.cu) pays a hand-off
// through L2 -- a store on one SM, a poll on another, 1.2-1.4 us -- for every
// level.  Here a thread owns a line and walks it row by row, a CTA owns a tile
// of TI x TJ lines, and a value reaches the other lines of the tile through
// shared memory; only values crossing a tile boundary go through L2, and a
// chain crosses N/TI + P/TJ of those.
//
// Time.  Line (i, j) of a tile makes its row t at step s = t + skew(i, j), the
// skews such that every dependency belongs to an earlier step.  A warp owns a
// patch of PI x PJ lines and all its lanes are at one step, so a value comes to
// the lines of the same patch by a shuffle.  Values for another patch go to
// that warp's inbox in shared memory, a ring of R steps [group][step][lane]
// filed under the step that reads them.  Whether a step's inputs are there is
// asked once per block of KS steps, not per step: a warp starts a block when
// its neighbours' step counters (prog) say that their part is done.  Rows
// before a line's start and its one row past the end are zero, and so are lines
// outside the grid, where the records hold zeros: rr - 0 * 0 leaves rr as it is,
// bit for bit.
//
// What sets the time (B200): a step of a patch, and the hand-off between tiles.
// A step is 115-120 cycles in two dimensions and FP64 (FP32 95), ~190-220 in
// three: the chain shuffle, multiply, K dependent subtracts, multiply, and the
// issue of the warp's ~32 instructions.  So a step's operands are read a step
// ahead, a block's inputs are asked for during the block before, a block whose
// lanes all have rows has no tests per row, and records lie in memory as the
// stages have them, one bulk copy per stage: 51 instructions and 240 cycles a
// step before that (FP64, 512^2; 377 cycles at 128^3).  A tile boundary costs
// 1.5-2.5 us: a store to L2, a poll, the inbox, and the rest of a block on both
// sides.  One call of the lower sweep (~25 us of it the fill and the host's wait),
// level-ordered / before / now: 128^3 7-point 546 / 175 / 152 us (FP32 517 / 135 /
// 123), 96^3 27-point 850 / 365 / 279, 512^2 5-point 1,145 / 147 / 109, 100^2
// 224 / 52 / 47.  Slower: blocks of 2 steps (512^2 144, 128^3 152-181), of 8 (128^3
// 190 with the former kernel), a counter by cp.async groups in place of the
// stages' mbarriers (the loader then waits for each copy), and results stored two
// rows at a time (512^2 177, 128^3 184).  Earlier forms on
// 512^2: lanes advancing independently 830 us; lanes in step with tagged slots
// polled and voted on per row 281.
//
// A CTA's warps:
//   compute  a thread per line: shuffles and inbox values, fold, publish.
//   fetch    several lanes per halo line (lines of neighbouring tiles that this
//            tile depends on), one row each: poll the NaN-boxed output vector in
//            L2 and file the values in the inboxes.  A poll takes ~1,000 cycles,
//            so the lanes bound the rate of rows (two dimensions: 4 lanes 160 us
//            at 512^2, 8 lanes 113, 16 lanes 109).  (One lane polling several
//            rows: its loads of one cache line wait for each other, ~500 cycles
//            each.)
//   load     a warp per compute warp, per stage of KL steps: its records with one
//            bulk copy, right-hand sides with cp.async, one mbarrier per stage.
//            (Records too by cp.async, a block at a time: 550 cycles a block, more
//            than the four steps they feed.)
// A value is filed only when its reader's counter shows the ring slot free.
// That cannot block: a warp waits for an earlier patch to be less than KS steps
// ahead, or for a later patch or one fed by the same halo line to be within R
// steps, and around any circle of such waits the steps lost exceed those gained
// (R > 2 KS + the largest distance in steps between a value and its reader).
// Records are the row's K = G E + 1 entry values, farthest first, and its
// inverted diagonal, padded to 16 bytes.
//
// Progress: tiles are claimed by an atomic ticket in an order in which every
// dependency points to the same or an earlier tile (lines shifted by `sk` per
// plane where a stencil reaches forward in the previous plane), so a CTA only
// waits for CTAs that run or have ended.  Every wait is bounded by itself, from
// the last row that came (MTLGPU_TIMEOUT): a long sweep is no long wait.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <type_traits>

#include "device.cuh"
#include "internal.h"
#include "line_tiles.h"
#include "tma.cuh"

namespace mtlgpu {

using namespace dev;

namespace {

constexpr int kBlock = 256;
constexpr int kMaxOff = 13;     // entries of a 27-point factor row
constexpr int kMinLine = 8;     // shortest line
constexpr int kMaxThreads = 512;

// The stencils: G groups of entries on other lines, farthest first, group g on
// the line PA planes and PB (shifted) lines back, with E places each.
template <int G, int E> struct Stencil;
template <> struct Stencil<1, 1> {  // 5-point, two dimensions
  __host__ __device__ static constexpr int PA(int) { return 0; }
  __host__ __device__ static constexpr int PB(int) { return 1; }
};
template <> struct Stencil<2, 1> {  // 7-point
  __host__ __device__ static constexpr int PA(int g) { return g == 0; }
  __host__ __device__ static constexpr int PB(int g) { return g == 1; }
};
template <> struct Stencil<1, 3> : Stencil<1, 1> {};  // 9-point, two dimensions
template <> struct Stencil<4, 3> {  // 27-point; lines shifted by one per plane
  __host__ __device__ static constexpr int PA(int g) { return g < 3; }
  __host__ __device__ static constexpr int PB(int g) { return g < 3 ? 2 - g : 1; }
};

template <int G, int E>
struct Shape : Stencil<G, E> {
  using S = Stencil<G, E>;
  static constexpr int kSteps = 4;                 // steps per block
  static constexpr int kLoad = E == 1 ? 8 : 4;     // steps per stage
  static constexpr int kRing = E == 1 ? 32 : 16;   // steps an inbox holds
  static constexpr int amax = G > 1 ? 1 : 0;       // planes a line depends on
  static constexpr int sk = G == 4 ? 1 : 0;        // lines shifted per plane
  static constexpr int hl = G == 4 ? 2 : 1;        // halo lines left of a tile
  static constexpr int fetch = G == 1 ? 16 : E == 1 ? 8 : 4;     // lanes per halo line
  static constexpr int PJ = amax ? 8 : 32, PI = 32 / PJ;  // a warp's patch
  static constexpr int newest = E == 3 ? -1 : 0;   // place of a group's last value
  static constexpr int s1 = 1 - newest;            // skew per line
  static constexpr int s2 = amax ? 1 - newest : 0; // and per plane (shifted lines)
  // Extra skew between patches: with one place per group a value is read
  // exactly kSteps steps after it was made, so its slot does not wrap inside
  // a block.
  static constexpr int X = E == 1 ? kSteps - 1 : 0;
  // step of row 0 of line (gi, gj) of a tile (three places: the step before it
  // takes row 0 of the lines it depends on)
  __host__ __device__ static constexpr int skew(int gi, int gj) {
    return gj * s1 + gi * s2 + (gj / PJ + gi / PI) * X + (E == 3 ? 1 : 0);
  }
  __host__ __device__ static constexpr int back(int g) { return newest + S::PA(g) * s2 + S::PB(g) * s1; }
  __host__ __device__ static constexpr int dist(int g) { return S::PA(g) * PJ + S::PB(g); }
  static constexpr int far = G == 4 ? 5 : 1;       // largest back(g)
  // steps between a value and its reader in the next patch: the smallest and
  // the largest, to the right, below, and below on the right
  __host__ __device__ static constexpr int min_back(int r) { return r == 2 ? 3 + 2 * X : 1 + X; }
  __host__ __device__ static constexpr int max_back(int r) { return far + (r == 2 ? 2 * X : X); }
  static constexpr bool diagonal = G == 4;         // patches meet at corners
};

// The stencil: G lines of dependencies (farthest first) with E places each.
struct LineShape {
  int n, B, P, NI, G, E;
  int mirrored;                  // an upper factor: x order is reversed row order
  int a[4], b[4];
};

struct LineArgs {
  int n, B, P, NI, TI, TJ, ntj, ntiles;
  int rec_bytes, stages;
  int rhs_stride;               // bytes of one line's ring of right-hand sides
  int blocks, stage;            // stages a warp's records fill, bytes of one
  int off_rec, off_rhs, off_lines, off_prog, off_halo, off_bar, smem;
  int compute_warps, fetch_warps, steps;
};

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double rsqrt_rn(double a) { return __ddiv_rn(1.0, __dsqrt_rn(a)); }
__device__ __forceinline__ float rsqrt_rn(float a) { return __fdiv_rn(1.f, __fsqrt_rn(a)); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

// Shared-memory words by address, with the orderings the step counters need.
__device__ __forceinline__ void sts(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void lds(unsigned a, double& v) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
}
__device__ __forceinline__ void lds(unsigned a, float& v) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ int ld_shared_acquire(unsigned a) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_release(unsigned a, int v) {
  asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// A record's values and diagonal (KR elements) from shared memory: 16 bytes per
// lane and 512 bytes.
template <typename T, int KR>
__device__ __forceinline__ void load_record(const unsigned char* s, T (&rec)[KR]) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int i = 0; i < KR; i += V) {
    T w[V];
    ld16(reinterpret_cast<const T*>(s + i / V * 512), w);
#pragma unroll
    for (int u = 0; u < V; u++)
      if (i + u < KR) rec[i + u] = w[u];
  }
}

// A record: the row's entries and its inverted diagonal, padded to 16 bytes.
template <typename T, int G, int E>
__host__ __device__ constexpr int rec_bytes() {
  return ((G * E + 2) * (int)sizeof(T) + 15) & ~15;
}

// UP: an upper factor, whose rows store their nearest entry first.
// IC0: not a sweep but IC(0)'s inverse diagonal (itl/pc/ic_0.hpp:136-186 as
// factor.cu has it): records hold a_mk and a_kk, and a row makes
//     out[k] = 1 / sqrt(a_kk - sum_m (a_mk out[m])^2)     (m ascending),
// the same dependencies with another fold; *pivot is set where that is no
// positive finite number.
template <typename T, int G, int E, bool UP, bool IC0>
__global__ void __launch_bounds__(kMaxThreads, 1)
    line_sweep_kernel(const __grid_constant__ LineArgs A, const unsigned char* __restrict__ recs,
                      const T* __restrict__ in, T* out, unsigned* ticket, int* err,
                      long long limit, const int* skip, int* pivot) {
  if (skip && ld_relaxed(skip)) return;
  using S = Shape<G, E>;
  constexpr int kTs = (int)sizeof(T), K = G * E + 1, KS = S::kSteps, R = S::kRing;
  constexpr int KL = S::kLoad;
  constexpr int kSlot = 32 * kTs;            // one step of one group of an inbox
  constexpr int kInbox = G * R * kSlot;      // one warp's inbox
  constexpr int kRow = 32 * rec_bytes<T, G, E>(), kStage = KL * kRow;  // records of a step, a stage
  constexpr int kNever = INT32_MAX / 2;
  constexpr int dir = UP ? -1 : 1;           // from a row to the next one in x order
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ int s_tile, s_done;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nlines = A.compute_warps * 32, npj = A.TJ / S::PJ;
  const unsigned sm0 = smem_u32(sm), prog = sm0 + A.off_prog, halo = sm0 + A.off_halo;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + A.off_bar);
  int2* lines = reinterpret_cast<int2*>(sm + A.off_lines);
  if (tid == 0) {
    s_tile = (int)atomicAdd(ticket, 1u);
    s_done = 0;
  }
  __syncthreads();
  const int trow = s_tile / A.ntj, I0 = trow * A.TI;
  const int J0 = (line_tile_col0(trow, A.TI, A.TJ, S::sk) + s_tile % A.ntj) * A.TJ;
  // first row (in x order) of the line at (gi, gj) of the tile, -1 outside the grid
  auto line_first = [&](int gi, int gj) {
    const int i = I0 + gi, j = J0 + gj - i * S::sk;
    return i < 0 || i >= A.NI || j < 0 || j >= A.P ? -1 : (i * A.P + j) * A.B;
  };
  auto skew_of = [&](int gi, int gj) { return S::skew(gi, gj); };
  // line (gi, gj)'s thread, and its inbox address of group g
  auto thread_of = [&](int gi, int gj) {
    return (gi / S::PI * npj + gj / S::PJ) * 32 + gi % S::PI * S::PJ + gj % S::PJ;
  };
  auto inbox_of = [&](int l, int g) {
    return sm0 + (l >> 5) * kInbox + g * R * kSlot + (l & 31) * kTs;
  };
  for (int i = tid; i < A.compute_warps * kInbox / 16; i += blockDim.x)
    reinterpret_cast<int4*>(sm)[i] = make_int4(0, 0, 0, 0);
  // a stage is there when its right-hand sides (32 lanes) and records (one) are
  for (int i = tid; i < A.compute_warps * A.stages; i += blockDim.x) mbar_init(full + i, 33);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  for (int i = tid; i < A.compute_warps * (1 + A.fetch_warps); i += blockDim.x)
    reinterpret_cast<int*>(sm + A.off_prog)[i] = 0;  // prog, then halo
  // this thread's line
  int li = 0, lj = 0, first = -1;
  if (tid < nlines) {
    const int patch = tid >> 5;
    li = patch / npj * S::PI + lane / S::PJ;
    lj = patch % npj * S::PJ + lane % S::PJ;
    first = line_first(li, lj);
    // for the loaders: its first step and its row (x order) at step 0
    lines[tid] = first >= 0 ? make_int2(skew_of(li, lj), first - skew_of(li, lj))
                            : make_int2(kNever, 0);
  }
  const bool work = __syncthreads_or(first >= 0);  // a tile may lie outside the grid
  const int smask = A.stages - 1;

  if (!work) {
  } else if (warp < A.compute_warps) {
    // ---- compute: one line per thread
    const int B = A.B, skew = skew_of(li, lj);
    // this lane's row at step s is s - lo; it has none when s - lo >= B (unsigned)
    const int lo = first < 0 ? kNever : skew;
    const unsigned char* rec_s = sm + A.off_rec + warp * A.stages * kStage + lane * 16;
    const unsigned char* rhs_s = sm + A.off_rhs + tid * A.rhs_stride;
    const unsigned char* box_s = sm + warp * kInbox + lane * kTs;
    T* op = out + (first < 0 ? 0 : (UP ? A.n - 1 - first : first)) - (long long)dir * skew;
    bool near[G];       // group g comes from a lane of this warp
    unsigned tgt[G];    // inbox of the line of another patch that takes this one as group g
    int tpos[G];        // slot of the value made at step 0 there
#pragma unroll
    for (int g = 0; g < G; g++) {
      near[g] = lane / S::PJ >= S::PA(g) && lane % S::PJ >= S::PB(g);
      const int ci = li + S::PA(g), cj = lj + S::PB(g);
      const bool other = ci / S::PI != li / S::PI || cj / S::PJ != lj / S::PJ;
      tgt[g] = 0;
      tpos[g] = 0;
      if (other && ci < A.TI && cj < A.TJ) {
        tgt[g] = inbox_of(thread_of(ci, cj), g);
        tpos[g] = (S::newest + skew_of(ci, cj) - skew) * kSlot;
      }
    }
    // What a block waits for, one condition per lane: *cptr >= s0 + cthr.
    unsigned cptr = prog + warp * 4;  // no condition: its own counter, at least 0
    int cthr = -kNever;
    {
      const int pi = warp / npj, pj = warp % npj, npi = A.TI / S::PI;
      const int r = lane % 3, up = lane < 3 ? 1 : -1;  // right, below, diagonal
      const int qi = pi - (r != 0) * up, qj = pj - (r != 1) * up;
      if (lane < 6 && (r != 2 || S::diagonal) && qi >= 0 && qj >= 0 && qi < npi && qj < npj) {
        cptr = prog + (qi * npj + qj) * 4;
        cthr = up > 0 ? KS - S::min_back(r) : KS + S::max_back(r) - R;
      } else if (lane >= 6 && lane < 6 + A.fetch_warps) {
        cptr = halo + (warp * A.fetch_warps + lane - 6) * 4;
        cthr = KS;
      }
    }
    T w[G][E], hist[S::far];
#pragma unroll
    for (int g = 0; g < G; g++)
#pragma unroll
      for (int x = 0; x < E; x++) w[g][x] = T(0);
#pragma unroll
    for (int x = 0; x < S::far; x++) hist[x] = T(0);
    // Blocks in which every lane has a row at every step: s0 in [in_lo, in_hi].
    const int in_lo = __reduce_max_sync(0xffffffffu, lo);
    const int in_hi = __reduce_min_sync(0xffffffffu, lo) + B - KS;
    unsigned long long* bar = full + warp * A.stages;
    // Whether block `s0`, whose records are in stage st, has its inputs.
    auto gate = [&](int s0, int st, unsigned phase) {
      const int c = ld_shared_acquire(cptr);
      const bool m = s0 % KL != 0 || mbar_test(bar + st, phase);
      return m & (c >= s0 + cthr);
    };
    // A step's operands, read a step ahead of their use: record (two of 27
    // points in FP64 don't fit the registers), right-hand side and inbox values.
    constexpr int RB = K * kTs > 64 ? 1 : 2;
    T rec[RB][K + 1], rhs[2], box[2][G];
    auto load_rec = [&](const unsigned char* p, int u) {
      load_record<T, K + 1>(p + u * kRow, rec[u % RB]);
    };
    auto load = [&](const unsigned char* rp, const unsigned char* vp, const unsigned char* bp,
                    int u) {
      if (RB == 2) load_rec(rp, u);
      rhs[u & 1] = *reinterpret_cast<const T*>(vp + u * kTs);
#pragma unroll
      for (int g = 0; g < G; g++)
        box[u & 1][g] = *reinterpret_cast<const volatile T*>(bp + (g * R + u) * kSlot);
    };
    bool dead = false, ahead = false;  // ahead: this block's gate was passed in the last one
    int st = 0;
    unsigned phase = 0;
    const unsigned char *rp = rec_s, *vp = rhs_s, *bp = box_s;
    // The steps of a block; INNER: every lane has a row.
    auto block = [&](auto inner, int s0) {
      constexpr bool INNER = decltype(inner)::value;
      const int t0 = s0 - lo;
      unsigned tb[G];
#pragma unroll
      for (int g = 0; g < G; g++)  // one place: no wrap inside the block
        tb[g] = E == 1 ? tgt[g] + ((tpos[g] + (unsigned)s0 * kSlot) & (R * kSlot - 1)) : tgt[g];
#pragma unroll
      for (int u = 0; u < KS; u++) {
        bool next = false;
        if (RB == 1) load_rec(rp, u);
        if (u < KS - 1) {
          load(rp, vp, bp, u + 1);
        } else {
          const int part = (s0 + KS) % KL;
          if (part == 0) st = (st + 1) & smask;
          rp = rec_s + st * kStage + part * kRow;
          vp = rhs_s + (st * KL + part) * kTs;
          bp = box_s + ((s0 + KS) & (R - 1)) * kSlot;
          if (ahead) load(rp, vp, bp, 0);
        }
        if (u == KS - 2) {
          const int nst = (st + 1) & smask;
          if ((s0 + KS) % KL == 0) phase ^= nst == 0;
          next = gate(s0 + KS, nst, phase);
        }
        T nw[G], rr = IC0 ? rec[u % RB][K] : rhs[u & 1];
#pragma unroll
        for (int g = 0; g < G; g++) {
          const T x = __shfl_up_sync(0xffffffffu, hist[S::back(g) - 1], S::dist(g));
          nw[g] = near[g] ? x : box[u & 1][g];
        }
        // one entry's contribution to the row
        auto fold = [&](T a, T wv) {
          const T d = mul_rn(a, wv);
          rr = sub_rn(rr, IC0 ? mul_rn(d, d) : d);
        };
        if (UP) fold(rec[u % RB][K - 1], hist[0]);
#pragma unroll
        for (int q = 0; q < G * E; q++) {
          // farthest line first, and on it the farthest place (index E - 1);
          // the reverse for UP
          const int k = UP ? G * E - 1 - q : q, g = k / E, x = E - 1 - k % E;
          fold(rec[u % RB][k], x == 0 ? nw[g] : w[g][x > 0 ? x - 1 : 0]);
        }
        if (!UP) fold(rec[u % RB][K - 1], hist[0]);
        const T sum = rr;
        rr = IC0 ? rsqrt_rn(rr) : mul_rn(rr, rec[u % RB][K]);
        const bool row = INNER || (unsigned)(t0 + u) < (unsigned)B;
#pragma unroll
        for (int x = S::far - 1; x > 0; x--) hist[x] = hist[x - 1];
        hist[0] = row ? rr : T(0);
        if (row) st_relaxed(op + dir * u, rr);
        if (IC0 && row && (!(sum > T(0)) || !isfinite(rr)))
          atomicCAS(pivot, 0, (int)MTLGPU_ZERO_PIVOT);
#pragma unroll
        for (int g = 0; g < G; g++) {
          if (tgt[g])
            sts(E == 1 ? tb[g] + u * kSlot
                       : tb[g] + ((tpos[g] + (unsigned)(s0 + u) * kSlot) & (R * kSlot - 1)), hist[0]);
#pragma unroll
          for (int x = E - 1; x > 0; x--) w[g][x] = w[g][x - 1];
          w[g][0] = nw[g];
        }
        if (u == KS - 2) {
          ahead = __all_sync(0xffffffffu, next) && s0 + KS < A.steps;
          __syncwarp();
        }
      }
      op += dir * KS;
      __syncwarp();
      if (lane == 0) st_shared_release(prog + warp * 4, s0 + KS);
    };
    for (int s0 = 0; s0 < A.steps; s0 += KS) {
      if (!ahead) {
        for (long long fails = 0; !__all_sync(0xffffffffu, gate(s0, st, phase));) {
          if (++fails >= limit ||
              ((fails & 1023) == 0 && __any_sync(0xffffffffu, ld_relaxed(err) != 0))) {
            dead = true;
            break;
          }
        }
        if (dead) break;
        __syncwarp();
        load(rp, vp, bp, 0);
      }
      if (s0 >= in_lo && s0 <= in_hi) block(std::true_type(), s0);
      else block(std::false_type(), s0);
    }
    if (dead && lane == 0) atomicCAS(err, 0, (int)MTLGPU_TIMEOUT);
    __syncwarp();
    if (lane == 0) {
      st_shared_release(prog + warp * 4, kNever);
      atomicAdd(&s_done, 1);
    }
  } else if (warp < A.compute_warps + A.fetch_warps) {
    // ---- fetch: S::fetch lanes per halo line (a row of lines above the tile,
    // then hl lines left of each of its rows), each polling one of its next rows
    const int fw = warp - A.compute_warps, sub = lane % S::fetch;
    const int h = (fw * 32 + lane) / S::fetch, top = S::amax * (A.TJ + S::hl);
    int gi = 0, gj = 0, hfirst = -1;
    if (h < top + A.TI * S::hl) {
      gi = h < top ? -1 : (h - top) / S::hl;
      gj = (h < top ? h : (h - top) % S::hl) - S::hl;
      hfirst = line_first(gi, gj);
    }
    unsigned tgt[G];
    int due[G], cw[G];  // step that reads row 0; its warp
    bool any = false;
#pragma unroll
    for (int g = 0; g < G; g++) {
      const int ci = gi + S::PA(g), cj = gj + S::PB(g);
      tgt[g] = 0;
      due[g] = 0;
      cw[g] = -1;
      if (hfirst >= 0 && ci >= 0 && cj >= 0 && ci < A.TI && cj < A.TJ && line_first(ci, cj) >= 0) {
        const int l = thread_of(ci, cj);
        tgt[g] = inbox_of(l, g);
        due[g] = S::newest + skew_of(ci, cj);
        cw[g] = l >> 5;
        any = true;
      }
    }
    const T* o = out + (any ? (UP ? A.n - 1 - hfirst : hfirst) : 0);
    // rows to file: the line's, and (three places) the zero past its end
    const int len = any ? A.B + (E == 3 ? 1 : 0) : 0, last = any ? A.B - 1 : 0;
    // the compute warps this warp's lines feed; the others never wait for it
    unsigned fed = 0;
#pragma unroll
    for (int g = 0; g < G; g++)
      if (cw[g] >= 0) fed |= 1u << cw[g];
    fed = __reduce_or_sync(0xffffffffu, fed);
    if (lane < A.compute_warps && !(fed >> lane & 1))
      st_shared_release(halo + (lane * A.fetch_warps + fw) * 4, kNever);
    int t = 0;
    bool begun = false;
    // polls: those since the last row filed
    for (long long polls = 0; polls < limit; ++polls) {
      const int row = t + sub;
      T v = ld_relaxed(o + (long long)dir * min(row, last));
      int lim = len;
#pragma unroll
      for (int g = 0; g < G; g++)
        if (cw[g] >= 0) lim = min(lim, ld_shared_acquire(prog + cw[g] * 4) + R - due[g]);
      if (row > last) v = T(0);
      // the rows that are there, up to the first gap
      const unsigned got = __ballot_sync(0xffffffffu, row < lim && !Box<T>::is(v)) >> (lane - sub);
      const int cnt = __ffs(~(got & ((1u << S::fetch) - 1))) - 1;
      if (sub < cnt) {
#pragma unroll
        for (int g = 0; g < G; g++)
          if (cw[g] >= 0) sts(tgt[g] + ((row + due[g]) & (R - 1)) * kSlot, v);
      }
      t += cnt;
      // the steps whose values from this warp's lines are all filed, per warp
      // (at first: those before the lines' row 0)
      const bool filed = __any_sync(0xffffffffu, cnt > 0);
      if (filed) polls = -1;
      if (!begun || filed) {
        begun = true;
        __syncwarp();
        for (unsigned m = fed; m; m &= m - 1) {
          const int c = __ffs(m) - 1;
          int ready = kNever;
#pragma unroll
          for (int g = 0; g < G; g++)
            if (cw[g] == c && t < len) ready = min(ready, t + due[g]);
          ready = __reduce_min_sync(0xffffffffu, ready);
          if (lane == 0) st_shared_release(halo + (c * A.fetch_warps + fw) * 4, ready);
        }
      }
      if (!__any_sync(0xffffffffu, t < len)) break;
      if (__any_sync(0xffffffffu, *(volatile int*)&s_done == A.compute_warps)) break;
    }
  } else {
    // ---- load: a warp per compute warp.  Its records are one bulk copy per
    // stage (they lie in memory as they do in a stage); right-hand sides of a line
    // are taken by KL lanes, and the lines a lane copies for stay in registers.
    constexpr int kIt = KL;
    const int cw = warp - A.compute_warps - A.fetch_warps, u = lane % KL;
    const int2* tab = lines + cw * 32;  // (first step, row at step 0)
    int2 vl[kIt];
#pragma unroll
    for (int i = 0; i < kIt; i++) {
      vl[i] = tab[lane / KL + i * (32 / KL)];
      vl[i].x -= u;
      vl[i].y += u;
    }
    const T* in0 = in + (UP ? A.n - 1 : 0);
    unsigned char* rhs_d = sm + A.off_rhs + (cw * 32 + lane / KL) * A.rhs_stride + u * kTs;
    unsigned char* rec_d = sm + A.off_rec + cw * A.stages * kStage;
    unsigned long long* bar = full + cw * A.stages;
    // the block of the patch's first row
    const int b0 = skew_of(cw / npj * S::PI, cw % npj * S::PJ) / KL;
    const unsigned char* rec0 =
        recs + (((long long)s_tile * A.compute_warps + cw) * A.blocks - b0) * kStage;
    bool stop = false;
    int blk = 0;
    for (; blk < A.steps / KL; blk++) {
      const int st = blk & smask, s0 = blk * KL;
      long long polls = 0;
      int at;  // the compute warp's step; kNever here: it gave up
      while (s0 + KL - (at = ld_shared_acquire(prog + cw * 4)) > A.stages * KL) {
        if (++polls >= limit || *(volatile int*)&s_done == A.compute_warps) {
          stop = true;
          break;
        }
        __nanosleep(20);
      }
      // A stage is filled again only once the warp has taken it: its barrier must
      // have completed the phase before.
      if (__any_sync(0xffffffffu, stop || at >= kNever)) break;
      if (lane == 0) {
        if ((unsigned)(blk - b0) < (unsigned)A.blocks) {
          mbar_arrive_expect_tx(bar + st, kStage);
          bulk_copy_g2s(rec_d + st * kStage, rec0 + (long long)blk * kStage, kStage, bar + st);
        } else {
          mbar_arrive(bar + st);
        }
      }
#pragma unroll
      for (int i = 0; i < (IC0 ? 0 : kIt); i++)
        if ((unsigned)(s0 - vl[i].x) < (unsigned)A.B)
          cp_async_ca<kTs>(rhs_d + i * (32 / KL) * A.rhs_stride + st * KL * kTs,
                           in0 + (long long)dir * (vl[i].y + s0));
      __syncwarp();
      mbar_arrive_cp_async(bar + st);
    }
    // Every copy has landed before the block ends, also one that gave up: copies
    // wait for nobody, so this has a bound of its own.
    cp_async_wait_all();
    const long long drain = limit > (1ll << 24) ? limit : (1ll << 24);
    for (int k = max(0, blk - A.stages); k < blk; k++)
      mbar_wait(bar + (k & smask), (unsigned)(k / A.stages) & 1u, drain);
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(ticket + 1, 1u) == (unsigned)A.ntiles - 1) {
      ticket[0] = 0;
      ticket[1] = 0;
      __threadfence();
    }
  }
}

// ---------------------------------------------------------------------------
// Analysis.

// Entry k (farthest first; k = G E: the predecessor) of row (i, j, t): whether
// its place is in the grid, and its distance.
__device__ __forceinline__ bool entry_of(const LineShape& S, int k, int i, int j, int t, int* d) {
  if (k == S.G * S.E) {
    *d = 1;
    return t >= 1;
  }
  const int g = k / S.E, e = S.E == 3 ? 1 - k % 3 : 0;
  *d = (S.a[g] * S.P + S.b[g]) * S.B + e;
  const int jj = j - S.b[g], tt = t - e;
  return i >= S.a[g] && jj >= 0 && jj < S.P && tt >= 0 && tt < S.B;
}

// Every row has exactly the stencil's entries that lie in the grid, in order.
__global__ void line_verify_kernel(LineShape S, const int32_t* __restrict__ rp,
                                   const int32_t* __restrict__ ci, int* bad) {
  const int K = S.G * S.E + 1;
  for (long long r = gtid(); r < S.n; r += gstride()) {
    if (ld_relaxed(bad)) return;
    const int x = S.mirrored ? S.n - 1 - (int)r : (int)r;
    const int t = x % S.B, j = x / S.B % S.P, i = x / S.B / S.P;
    int q = rp[r];
    const int end = rp[r + 1];
    for (int kk = 0; kk < K; kk++) {
      int d;
      if (!entry_of(S, S.mirrored ? K - 1 - kk : kk, i, j, t, &d)) continue;
      if (q < end && ci[q] == (int)r) q++;  // a diagonal stored first
      if (q >= end || (S.mirrored ? ci[q] - (int)r : (int)r - ci[q]) != d) {
        st_relaxed(bad, 1);
        return;
      }
      q++;
    }
    if (q < end && ci[q] == (int)r) q++;
    if (q != end) {
      st_relaxed(bad, 1);
      return;
    }
  }
}

// Records: the entries' values farthest first (outside the grid: zero), the
// inverted diagonal (1 for a unit diagonal), zero padding; row x's where the
// sweep's stages have them: [tile][warp][stage][step][16 bytes][lane].  `round`
// gives double records the float values.
template <typename T, int G, int E>
__global__ void line_fill_kernel(const __grid_constant__ LineShape L,
                                 const __grid_constant__ LineArgs A,
                                 const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                 const double* __restrict__ v, bool unit, bool round,
                                 unsigned char* __restrict__ rec) {
  using S = Shape<G, E>;
  constexpr int K = G * E + 1, V = 16 / (int)sizeof(T), KL = S::kLoad;
  constexpr int kPpr = rec_bytes<T, G, E>() / 16;
  for (long long x = gtid(); x < L.n; x += gstride()) {
    const int r = L.mirrored ? L.n - 1 - (int)x : (int)x;
    const int t = (int)(x % L.B), j = (int)(x / L.B % L.P), i = (int)(x / L.B / L.P);
    const int js = j + i * S::sk, gi = i % A.TI, gj = js % A.TJ;
    const int pi = gi / S::PI, pj = gj / S::PJ, npj = A.TJ / S::PJ;
    const int step = t + S::skew(gi, gj), b0 = S::skew(pi * S::PI, pj * S::PJ) / KL;
    const long long warp =
        line_tile_of(i, js, A.TI, A.TJ, S::sk, A.ntj) * A.compute_warps + pi * npj + pj;
    const int lane = gi % S::PI * S::PJ + gj % S::PJ;
    unsigned char* o = rec + (((warp * A.blocks + step / KL - b0) * KL + step % KL) * kPpr * 32 + lane) * 16;
    int q = rp[r];
    T w[kPpr * V];
    w[K] = T(1);
    auto val = [&](int at) { return round ? (T)(float)v[at] : (T)v[at]; };
    if (!unit) w[K] = val(ci[q] == r ? q : rp[r + 1] - 1);
    if (!unit && ci[q] == r) q++;
#pragma unroll
    for (int kk = 0; kk < K; kk++) {
      int d;
      if (L.mirrored)
        w[K - 1 - kk] = entry_of(L, K - 1 - kk, i, j, t, &d) ? val(q++) : T(0);
      else
        w[kk] = entry_of(L, kk, i, j, t, &d) ? val(q++) : T(0);
    }
#pragma unroll
    for (int k = K + 1; k < kPpr * V; k++) w[k] = T(0);
#pragma unroll
    for (int c = 0; c < kPpr; c++) {
      T e[V];
#pragma unroll
      for (int u = 0; u < V; u++) e[u] = w[c * V + u];
      st16(reinterpret_cast<T*>(o + c * 512), e);
    }
  }
}

int round_div(int x, int y) { return (x + y / 2) / y; }

// The stencil whose distances (largest first, the last one 1) are d, for line
// length B and P lines per plane; false when they are none of the supported
// ones.
bool line_stencil(const int* d, int nd, int B, int P, LineShape* S) {
  S->B = B;
  S->P = P;
  S->G = 0;
  S->E = 0;
  for (int k = 0; k < nd - 1;) {
    const int q = round_div(d[k], B), e = d[k] - q * B;
    const int a = round_div(q, P), b = q - a * P;
    // three places e = 1, 0, -1, or the place itself
    int E = 1;
    if (e == 1) {
      if (k + 2 >= nd - 1 || d[k + 1] != q * B || d[k + 2] != q * B - 1) return false;
      E = 3;
    } else if (e != 0) {
      return false;
    }
    if (a < 0 || a > 1 || b < -1 || b > 1 || (a == 0 && b != 1)) return false;
    if (S->G == 4 || (S->E && S->E != E)) return false;
    S->E = E;
    S->a[S->G] = a;
    S->b[S->G] = b;
    S->G++;
    k += E;
  }
  // kernels exist for 5-, 7-, 9- and 27-point
  auto is = [&](int g, int a, int b) { return S->a[g] == a && S->b[g] == b; };
  if (S->G == 1) return is(0, 0, 1);
  if (S->E == 1) return S->G == 2 && is(0, 1, 0) && is(1, 0, 1);
  return S->G == 4 && is(0, 1, 1) && is(1, 1, 0) && is(2, 1, -1) && is(3, 0, 1);
}

int smem_limit(Ctx* ctx) {
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) !=
      cudaSuccess)
    v = 0;
  return v - 1024;
}

// Tile, rings and shared-memory layout for element size ts; false: no tile fits.
template <int G, int E>
bool line_layout_t(Ctx* ctx, const LineShape& L, int ts, LineArgs* A) {
  using S = Shape<G, E>;
  std::memset(A, 0, sizeof(*A));
  A->n = L.n;
  A->B = L.B;
  A->P = L.P;
  A->NI = L.NI;
  A->rec_bytes = ts == 8 ? rec_bytes<double, G, E>() : rec_bytes<float, G, E>();
  A->stage = S::kLoad * 32 * A->rec_bytes;
  // Three dimensions: patches one above the other, two of them, or four where
  // two make more tiles than the chip has SMs (a CTA per SM).  A call of the
  // lower sweep with 8 x 8 / 16 x 8 lines (33^3, 96^3, 128^3 7-point, FP64: 55 / 60,
  // 104 / 109, 157 / 152 us; FP32 49 / 52, 97 / 97, 136 / 124; 47^3 27-point FP32
  // 110 / 119; 8 x 16 and 4 x 8 lines lost to both).  27 points in FP64: one patch,
  // 47^3 124, 96^3 279 us (two: 132 / 300, four: 145 / 301).  Two dimensions: one
  // patch.  Stages: four where they fit, else two (16 x 8 lines in FP64: the same
  // time).
  A->TJ = S::PJ;
  A->TI = !S::amax ? 1 : G == 4 && ts == 8 ? 4 : 8;
  auto tiles = [&] { return line_tile_count(L.P, L.NI, A->TI, A->TJ, S::sk); };
  if (A->TI == 8 && tiles() > ctx->num_sms) A->TI = 16;
  const int limit = smem_limit(ctx);
  for (A->stages = 4;; A->stages == 4 ? A->stages = 2 : (A->stages = 4, A->TI /= 2)) {
    if (A->TI < S::PI) return false;
    const int lines = A->TI * A->TJ, rows = A->stages * S::kLoad;
    const int halo = S::amax * (A->TJ + S::hl) + A->TI * S::hl;
    A->compute_warps = lines / 32;
    A->fetch_warps = (halo * S::fetch + 31) / 32;
    A->rhs_stride = (rows + 1) * ts;  // the lanes' accesses spread over the banks
    int o = lines * G * S::kRing * ts;  // inboxes
    A->off_rec = o;
    o += lines * rows * A->rec_bytes;
    A->off_rhs = o;
    o = (o + lines * A->rhs_stride + 7) & ~7;
    A->off_bar = o;
    o += A->compute_warps * A->stages * 8;
    A->off_lines = o;
    o += lines * 8;
    A->off_prog = o;
    o += A->compute_warps * 4;
    A->off_halo = o;
    o += A->compute_warps * A->fetch_warps * 4;
    A->smem = o;
    if (o <= limit && (2 * A->compute_warps + A->fetch_warps) * 32 <= kMaxThreads) break;
  }
  if (tiles() > INT32_MAX) return false;
  A->ntj = line_tile_cols(L.P, L.NI, A->TI, A->TJ, S::sk);
  A->ntiles = (int)tiles();
  // the last line's last step makes the zero row past its end
  const int skew = (A->TJ - 1) * S::s1 + (A->TI - 1) * S::s2 +
                   (A->TJ / S::PJ + A->TI / S::PI - 2) * S::X + 1;
  A->steps = (skew + L.B + 1 + S::kLoad - 1) / S::kLoad * S::kLoad;
  // from the stage of a patch's first row to that of its last
  A->blocks = (S::kLoad - 1 + S::skew(S::PI - 1, S::PJ - 1) - S::skew(0, 0) + L.B - 1) / S::kLoad + 1;
  return true;
}
size_t record_bytes(const LineArgs& A) {
  return (size_t)A.ntiles * A.compute_warps * A.blocks * A.stage;
}
bool line_layout(Ctx* ctx, const LineShape& L, int ts, LineArgs* A) {
  const bool fits =
      L.E == 1 ? (L.G == 1 ? line_layout_t<1, 1>(ctx, L, ts, A) : line_layout_t<2, 1>(ctx, L, ts, A))
               : (L.G == 1 ? line_layout_t<1, 3>(ctx, L, ts, A) : line_layout_t<4, 3>(ctx, L, ts, A));
  if (!fits) return false;
  const long long own = (long long)L.n * A->rec_bytes, padded = (long long)record_bytes(*A);
  if (line_records_fit(own, padded, 0)) return true;
  size_t free_bytes = 0;  // asking for the device's memory takes up to milliseconds
  if (!ctx->device_bytes &&
      cudaMemGetInfo(&free_bytes, &ctx->device_bytes) != cudaSuccess)
    cudaGetLastError();
  return line_records_fit(own, padded, (long long)ctx->device_bytes);
}

template <typename T>
using LineKernel = void (*)(const LineArgs, const unsigned char*, const T*, T*, unsigned*, int*,
                            long long, const int*, int*);

template <typename T>
LineKernel<T> line_kernel(const LineShape& S) {
  if (S.E == 1 && S.G == 1)
    return S.mirrored ? line_sweep_kernel<T, 1, 1, true, false> : line_sweep_kernel<T, 1, 1, false, false>;
  if (S.E == 1)
    return S.mirrored ? line_sweep_kernel<T, 2, 1, true, false> : line_sweep_kernel<T, 2, 1, false, false>;
  if (S.G == 1)
    return S.mirrored ? line_sweep_kernel<T, 1, 3, true, false> : line_sweep_kernel<T, 1, 3, false, false>;
  return S.mirrored ? line_sweep_kernel<T, 4, 3, true, false> : line_sweep_kernel<T, 4, 3, false, false>;
}
LineKernel<double> line_ic0_kernel(const LineShape& S) {
  if (S.E == 1)
    return S.G == 1 ? line_sweep_kernel<double, 1, 1, false, true>
                    : line_sweep_kernel<double, 2, 1, false, true>;
  return S.G == 1 ? line_sweep_kernel<double, 1, 3, false, true>
                  : line_sweep_kernel<double, 4, 3, false, true>;
}

template <typename T>
mtlgpu_status line_launch(Ctx* ctx, LineKernel<T> kernel, const LineArgs& A, const void* rec,
                          const T* in, T* out, unsigned* ticket, const int* skip, int* pivot) {
  ctx->launches++;
  kernel<<<A.ntiles, (2 * A.compute_warps + A.fetch_warps) * 32, A.smem, ctx->stream>>>(
      A, static_cast<const unsigned char*>(rec), in, out, ticket, ctx->d_error, ctx->spin_limit,
      skip, pivot);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return MTLGPU_OK;
}

int line_grid(Ctx* ctx, int n) {
  return (int)std::min<long long>(((long long)n + kBlock - 1) / kBlock, ctx->num_sms * 8ll);
}

template <typename T>
void line_fill_launch(Ctx* ctx, const LineShape& S, const LineArgs& A, const int32_t* rp,
                      const int32_t* ci, const double* v, bool unit, bool round,
                      unsigned char* rec) {
  const int grid = line_grid(ctx, S.n);
#define MTLGPU_LF(G, E) \
  line_fill_kernel<T, G, E><<<grid, kBlock, 0, ctx->stream>>>(S, A, rp, ci, v, unit, round, rec)
  if (S.E == 1) {
    if (S.G == 1) MTLGPU_LF(1, 1); else MTLGPU_LF(2, 1);
  } else {
    if (S.G == 1) MTLGPU_LF(1, 3); else MTLGPU_LF(4, 3);
  }
#undef MTLGPU_LF
}

// Whether every row has S's entries (flag: one device int, 4 bytes of scratch).
mtlgpu_status line_verify(Ctx* ctx, const LineShape& S, const int32_t* d_rp, const int32_t* d_ci,
                          int* flag, bool* ok) {
  int bad = 0;
  MTLGPU_TRY_CUDA(ctx, cudaMemsetAsync(flag, 0, sizeof(int), ctx->stream));
  line_verify_kernel<<<line_grid(ctx, S.n), kBlock, 0, ctx->stream>>>(S, d_rp, d_ci, flag);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  MTLGPU_TRY_CUDA(ctx, cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost,
                                       ctx->stream));
  MTLGPU_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  *ok = bad == 0;
  return MTLGPU_OK;
}

// The stencil of the pattern (rows of one triangle, stored diagonals
// ignored), if it is one.
mtlgpu_status line_find(Ctx* ctx, LineShape* S, const int32_t* d_rp, const int32_t* d_ci, int* d_s,
                        bool* found) {
  *found = false;
  const int n = S->n;
  int off[32], cnt = 0, d[kMaxOff], nd = 0;
  MTLGPU_TRY(sample_offsets(ctx, n, d_rp, d_ci, 0, off, &cnt));
  if (cnt > kMaxOff + 1) return MTLGPU_OK;
  for (int k = 0; k < cnt; k++)
    if (off[k] && nd < kMaxOff) d[nd++] = std::abs(off[k]);
  std::sort(d, d + nd, [](int x, int y) { return x > y; });
  if (nd < 2 || d[nd - 1] != 1) return MTLGPU_OK;
  // candidates: B a distance, P a number of lines at another distance, or (two
  // dimensions) all lines in one plane
  for (int kb = nd - 2; kb >= 0; kb--) {
    const int B = d[kb];
    if (B < kMinLine || n % B) continue;
    const int lines = n / B;
    for (int kp = kb - 1; kp >= -1; kp--) {
      const int lp = kp >= 0 ? round_div(d[kp], B) : lines;
      if (lp < 2 || lp > lines || lines % lp || !line_stencil(d, nd, B, lp, S)) continue;
      S->NI = lines / lp;
      MTLGPU_TRY(line_verify(ctx, *S, d_rp, d_ci, d_s, found));
      if (*found) return MTLGPU_OK;
    }
  }
  return MTLGPU_OK;
}

}  // namespace

struct LinePlan {
  LineShape shape;
  LineArgs args[2];              // per precision (0: double, 1: float)
  void* d_rec[2] = {nullptr, nullptr};  // records, made by line_plan_fill
  unsigned* d_ticket = nullptr;
};

// Gives P its grid-line form (without records yet) when the pattern is that of
// a grid stencil; `like` (may be null): the other triangle's plan, whose grid
// is tried instead of searching.  P's n, nnz_off and reverse are set.  Outside
// any stream capture.
mtlgpu_status line_plan_detect(Ctx* ctx, SweepPlan* P, const SweepPlan* like, const int32_t* d_rp,
                               const int32_t* d_ci) {
  line_plan_free(ctx, P);
  if (P->n == 0 || P->nnz_off == 0 || ctx->part_sweeps != 2 || (like && !like->line))
    return MTLGPU_OK;
  int* d_s = nullptr;
  MTLGPU_TRY(dalloc(ctx, &d_s, 1));
  LineShape S{};
  bool found = false;
  mtlgpu_status st = MTLGPU_OK;
  if (like) {
    S = like->line->shape;
    S.mirrored = P->reverse;
    st = line_verify(ctx, S, d_rp, d_ci, d_s, &found);
  } else {
    S.n = P->n;
    S.mirrored = P->reverse;
    st = line_find(ctx, &S, d_rp, d_ci, d_s, &found);
  }
  dfree(ctx, d_s);
  MTLGPU_TRY(st);
  LineArgs A[2];
  if (!found || !line_layout(ctx, S, 8, &A[0]) || !line_layout(ctx, S, 4, &A[1])) return MTLGPU_OK;
  LinePlan* L = new LinePlan();
  P->line = L;
  // Row t of line j of plane i is of level t + j + i, with three places
  // t + 2 j + 4 i (a row waits for the next place of the next line of the plane
  // before).
  const int step = S.E == 3 ? 2 : 1;
  P->n_levels = S.B + step * (S.P - 1) + step * step * (S.NI - 1);
  L->shape = S;
  L->args[0] = A[0];
  L->args[1] = A[1];
  st = dalloc(ctx, &L->d_ticket, 2);
  cudaError_t e = cudaSuccess;
  if (st == MTLGPU_OK) e = cudaMemsetAsync(L->d_ticket, 0, 8, ctx->stream);
  const int smem = smem_limit(ctx);
  for (const void* k : {reinterpret_cast<const void*>(line_kernel<double>(S)),
                        reinterpret_cast<const void*>(line_kernel<float>(S)),
                        reinterpret_cast<const void*>(line_ic0_kernel(S))})
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) st = set_cuda_error(ctx, e, "line plan");
  if (st != MTLGPU_OK) line_plan_free(ctx, P);
  return st;
}

// The records of one precision from the factor's values; `round`: double
// records hold the float values (FP32 factors).
mtlgpu_status line_plan_fill(Ctx* ctx, SweepPlan* P, int prec, const int32_t* d_rp,
                             const int32_t* d_ci, const double* d_v, bool round) {
  LinePlan& L = *P->line;
  const LineShape& S = L.shape;
  const LineArgs& A = L.args[prec];
  unsigned char* rec = static_cast<unsigned char*>(L.d_rec[prec]);
  if (!rec) {
    MTLGPU_TRY(dalloc(ctx, &rec, record_bytes(A)));
    L.d_rec[prec] = rec;
  }
  if (prec)
    line_fill_launch<float>(ctx, S, A, d_rp, d_ci, d_v, P->unit_diag, true, rec);
  else
    line_fill_launch<double>(ctx, S, A, d_rp, d_ci, d_v, P->unit_diag, round, rec);
  MTLGPU_TRY_CUDA(ctx, cudaGetLastError());
  return MTLGPU_OK;
}

// IC(0)'s inverse diagonal into d_inv from L's pattern carrying a_mk, a_kk
// last (factor.cu).  Uses and then drops L's double records.
mtlgpu_status line_ic0_inverse(Ctx* ctx, SweepPlan* L, const int32_t* d_rp, const int32_t* d_ci,
                               const double* d_a, double* d_inv, int* d_pivot) {
  MTLGPU_TRY(line_plan_fill(ctx, L, 0, d_rp, d_ci, d_a, false));
  MTLGPU_TRY(fill_sentinel<double>(ctx, d_inv, L->n));
  LinePlan& P = *L->line;
  MTLGPU_TRY(line_launch<double>(ctx, line_ic0_kernel(P.shape), P.args[0], P.d_rec[0], nullptr,
                                 d_inv, P.d_ticket, nullptr, d_pivot));
  dfree(ctx, P.d_rec[0]);
  return MTLGPU_OK;
}

void line_plan_free(Ctx* ctx, SweepPlan* P) {
  if (!P->line) return;
  for (void*& r : P->line->d_rec) dfree(ctx, r);
  dfree(ctx, P->line->d_ticket);
  delete P->line;
  P->line = nullptr;
}

bool line_records_ready(const SweepPlan& P, int prec) { return P.line && P.line->d_rec[prec]; }

template <typename T>
mtlgpu_status line_sweep_launch(Ctx* ctx, const SweepPlan& P, const T* in, T* out,
                                const int* skip) {
  const LinePlan& L = *P.line;
  const int prec = sizeof(T) == 8 ? 0 : 1;
  return line_launch<T>(ctx, line_kernel<T>(L.shape), L.args[prec], L.d_rec[prec], in, out,
                        L.d_ticket, skip, nullptr);
}

template mtlgpu_status line_sweep_launch<double>(Ctx*, const SweepPlan&, const double*, double*,
                                                 const int*);
template mtlgpu_status line_sweep_launch<float>(Ctx*, const SweepPlan&, const float*, float*,
                                                const int*);

}  // namespace mtlgpu
