// dustb_deposit.cuh -- FP64 stencil deposits combined per cell inside a warp.
//
// A particle's deposit is 27 cells (9 in 2-D) times up to four values.  One FP64 atomic per
// particle, cell and value is bound by the L2's atomic rate (0.17 T atomics/s: 2.6-2.9 ms for
// each 3-D deposit of 4.2 M particles at 16 per cell).  Here a warp takes 32 consecutive
// particles at a time: every lane forms one particle's weights and values and stages them in
// the warp's shared memory in ascending order of the anchor cells; then the lanes become the
// 27 cells of one stencil and walk the particles of one anchor cell after the other, summing
// in registers.  When the next anchor is the next cell along x, two thirds of the window carry
// over by a shuffle and only the column left behind is added to the field (9 lanes x values
// atomics per cell instead of 27 per particle).  Rows in cell order need about 2 atomics per
// particle instead of 108; rows in no order make groups of one particle, whose atomics are no
// more than before and land on three consecutive cells per row.  A batch adds lane by lane
// instead, one atomic per particle, cell and value, where that is faster or where a value is not
// finite (deposit_particles, deposit_clouds say when).
//
// A contribution differs from the one-thread-per-particle form's by its rounding: the weight is
// ((wz f) wy) wx with the factor f second instead of ((wz wy) f) wx, and the windows add weight
// times value by a fused multiply-add where the lane-by-lane form rounds the product first.  With
// three roundings of each weight and one of the product, the two forms differ by at most
// 4 eps = 2^-50 of the contribution.
//
// 4.2 M particles at 16 per cell (64^3 cells, 5 CTAs per SM), the mean of the eight stages after
// a sort: Q/P 2.88 -> 0.35 ms (with the centre mass), operator 2.59 -> 0.41, gather-kick 2.63 ->
// 0.49.  What bounds it now is instruction issue and its latencies (IPC 2.0, 38 warp
// instructions per particle in Q/P: about 9 to form and stage a particle, 10 to sum it, the
// rest the changes of cell), no longer atomics (L2 at 25 %).  Measured and not kept: nine lanes
// per stream with three x columns and all values in registers (0.40 ms Q/P: the streams'
// flushes diverge); six CTAs per SM (80 registers, spilled: 4 % slower).
#pragma once

#include "dustb_common.cuh"

namespace dustb {

constexpr int kDepWarps = 4;                     // warps per CTA of the depositing kernels
constexpr unsigned kNoCell = 0xffffffffu;

// one warp's staged batch: up to four values per particle, the x weights (rows 0-2) and the
// products of y and z weights with the particle's factor (rows 3-11: 3 + 3 c + b).  33 columns:
// the rows the lanes of one load read lie in different banks
struct alignas(16) WarpStage {
  double q[32][4];              // (first: its 16-byte loads; the size is a multiple of 16)
  double w[12][33];
  long long kb[32];             // the anchor cell's field index
  unsigned key[32];             // the anchor cell (ascending)
  __device__ __forceinline__ void put(int at, const double wx[3], const double wy[3],
                                      const double wz[3], double fac, const double v[4],
                                      unsigned k, long long at_k) {
#pragma unroll
    for (int a = 0; a < 3; ++a) w[a][at] = wx[a];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double f = wz[c] * fac;
#pragma unroll
      for (int b = 0; b < 3; ++b) w[3 + 3 * c + b][at] = f * wy[b];
    }
    *(double2 *)&q[at][0] = make_double2(v[0], v[1]);
    *(double2 *)&q[at][2] = make_double2(v[2], v[3]);
    key[at] = k;
    kb[at] = at_k;
  }
};
static_assert(sizeof(WarpStage) % 16 == 0, "the stages of a CTA follow one another");

// consecutive batches of 32 particles a warp takes: enough that the cells at a warp's ends are
// shared, few enough for several waves of CTAs
inline int dep_batches(long long n) {
  const long long per = n / (32LL * 148 * 64);
  return per < 1 ? 1 : (per > 8 ? 8 : (int)per);
}
inline unsigned dep_blocks(long long n, int nb) {
  const long long per = 32LL * kDepWarps * nb;
  return (unsigned)((n + per - 1) / per);
}

// the place of this lane's particle among the warp's live ones in ascending key order (equal
// keys by lane; a lane without a particle holds kNoCell); all lanes of the warp take part
__device__ __forceinline__ int warp_rank(unsigned key, bool live) {
  const int lane = threadIdx.x & 31;
  const unsigned up = __shfl_up_sync(0xffffffffu, key, 1);
  if (__all_sync(0xffffffffu, lane == 0 || up <= key)) return lane;
  const unsigned below = (1u << lane) - 1u;
  int rank = 0, base = 0;
  unsigned rem = __ballot_sync(0xffffffffu, live);
  while (rem) {
    const bool mine = (rem >> lane) & 1u;
    const unsigned k = __reduce_min_sync(0xffffffffu, mine ? key : kNoCell);
    const unsigned grp = __ballot_sync(0xffffffffu, mine && key == k);
    if (mine && key == k) rank = base + __popc(grp & below);
    base += __popc(grp);
    rem &= ~grp;
  }
  return rank;
}

// NV values per cell; ONE: the first is the weight itself, the others the weight times q[0],
// q[1], ...
// at(k): the field address (variable 0) of this lane's window cell about the anchor with field
// index k, null if no block owns it; variables vs apart.  CEN: lane 27, which has no window
// cell, sums q[3] of the anchor cell's particles instead
template <int NV, bool ONE, bool CEN = false>
struct CellDeposit {
  static constexpr int NQ = NV - (ONE ? 1 : 0);
  double acc[NV];
  long long base;               // the field index of the current anchor cell
  unsigned cur;                 // the current anchor cell (kNoCell: none)
  int a, b, c;                  // this lane's cell of the window, -1..1 each
  bool on, centre;

  // lane = 9 (a + 1) + 3 (c + 1) + b + 1: a column is nine consecutive lanes
  __device__ __forceinline__ void init(bool three_d) {
    const int lane = threadIdx.x & 31, l = lane < 27 ? lane : 0;
    const int r = l % 9;
    a = l / 9 - 1; c = r / 3 - 1; b = r % 3 - 1;
    on = lane < 27 && (three_d || c == 0);
    centre = CEN && lane == 27;
    cur = kNoCell;
    base = 0;
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  }
  template <typename At>
  __device__ __forceinline__ void put(bool who, long long vs, At &&at) {
    if (!(who || centre)) return;
    double *t = at(base);
    if (!t) return;
#pragma unroll
    for (int v = 0; v < NV; ++v)
      if (acc[v] != 0.0 && (v == 0 || !centre)) atomicAdd(t + v * vs, acc[v]);
  }
  template <typename At>
  __device__ __forceinline__ void flush(long long vs, At &&at) {
    if (cur != kNoCell) put(on, vs, at);
    cur = kNoCell;
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  }
  template <typename At>
  __device__ __forceinline__ void move_to(unsigned k, long long kb, long long vs, At &&at) {
    if (k == cur) return;
    if (cur != kNoCell && k == cur + 1) {
      // the next cell of the row (a row's last padded cell is no anchor, so cur + 1 is never
      // the next row's): column 0 is finished, columns 1 and 2 become 0 and 1
      const int lane = threadIdx.x & 31;
      put(on && lane < 9, vs, at);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double y = __shfl_down_sync(0xffffffffu, acc[v], 9);
        acc[v] = lane < 18 ? y : 0.0;
      }
    } else {
      flush(vs, at);
    }
    cur = k;
    base = kb;
  }
  // the n staged particles of the batch, whose values are all finite (the zero weights of a
  // stencil then add nothing)
  template <typename At>
  __device__ __forceinline__ void walk(const WarpStage &s, int n, long long vs, At &&at) {
    const int lane = threadIdx.x & 31;
    const unsigned key = lane < n ? s.key[lane] : kNoCell;
    const double *wx = s.w[a + 1], *wyz = s.w[3 + 3 * (c + 1) + b + 1];
    int lo = 0;
    while (lo < n) {
      const unsigned k = __shfl_sync(0xffffffffu, key, lo);
      const int hi = lo + __popc(__ballot_sync(0xffffffffu, key == k));
      move_to(k, s.kb[lo], vs, at);
#pragma unroll 4
      for (int p = lo; p < hi; ++p) {
        const double w = wyz[p] * wx[p];
        if (ONE) acc[0] += centre ? s.q[p][3] : w;
#pragma unroll
        for (int v = 0; v < NQ; ++v)
          acc[v + (ONE ? 1 : 0)] = __fma_rn(w, s.q[p][v], acc[v + (ONE ? 1 : 0)]);
      }
      lo = hi;
    }
  }
};

}  // namespace dustb
