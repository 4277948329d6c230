// dustb_deposit.cuh -- FP64 stencil deposits combined per cell inside a warp.
//
// A particle's deposit is 27 cells (9 in 2-D) times up to four values.  One FP64 atomic per
// particle, cell and value is bound by the L2's atomic rate (the three 3-D deposits of a stage
// of 4.2 M particles at 16 per cell took 2.6-2.9 ms each, 0.17 T atomics/s).  Here a warp takes
// 32 consecutive particles at a time: every lane forms its own particle's weights and values
// and stages them in the warp's shared memory, then the lanes become the 27 cells of one
// stencil and walk the particles that share an anchor cell, summing in registers.  The groups
// of a batch go in ascending cell order; when the next group is the next cell along x, two
// thirds of the window carry over by a shuffle and only the column left behind is added to the
// field (9 lanes x values atomics per cell instead of 27 per particle).  Rows in cell order
// need about 2 atomics per particle instead of 108; rows in no order make groups of one
// particle, whose atomics are no more than before and land on three consecutive cells per
// row.  The products are those of the one-thread-per-particle form; only the order of the
// sums differs.
#pragma once

#include "dustb_common.cuh"

namespace dustb {

constexpr int kDepWarps = 4;                     // warps per CTA of the depositing kernels
constexpr unsigned kNoCell = 0xffffffffu;

// one warp's staged batch: the weights (x, y, z: rows 0-2, 3-5, 6-8; 33 columns, so that the
// three rows the lanes of one load read lie in different banks) and four values per particle
struct alignas(16) WarpStage {
  double q[32][4];              // (first: its 16-byte loads; the struct's size is padded to 16)
  double w[9][33];
  __device__ __forceinline__ void put(int lane, const double wx[3], const double wy[3],
                                      const double wz[3], double q0, double q1, double q2,
                                      double q3) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      w[a][lane] = wx[a];
      w[3 + a][lane] = wy[a];
      w[6 + a][lane] = wz[a];
    }
    *(double2 *)&q[lane][0] = make_double2(q0, q1);
    *(double2 *)&q[lane][2] = make_double2(q2, q3);
  }
};

// consecutive batches of 32 particles a warp takes: enough that the cells at a batch's ends
// are shared, few enough that small sets still give every SM 32 warps
inline int dep_batches(long long n) {
  const long long per = n / (32LL * 148 * 32);
  return per < 1 ? 1 : (per > 8 ? 8 : (int)per);
}
inline unsigned dep_blocks(long long n, int nb) {
  const long long per = 32LL * kDepWarps * nb;
  return (unsigned)((n + per - 1) / per);
}

// NV values per cell.  FAC: q[0] is a factor of the weights; ONE: the first value is the weight
// itself, the others the weight times q[FAC], q[FAC + 1], ...
template <int NV, bool FAC, bool ONE>
struct CellDeposit {
  double acc[NV];
  double *f;                    // variable 0 of the deposit
  long long vs;                 // its stride per variable
  long long base;               // the field index of the current anchor cell
  unsigned cur;                 // the current anchor cell (kNoCell: none)
  int ra, rb, rc, off;          // this lane's weights' rows and its cell's offset
  bool on;

  __device__ __forceinline__ void init(double *field, const Ind &d) {
    const int lane = threadIdx.x & 31;
    const int l = lane < 27 ? lane : 0;
    const int a = l / 9, r = l - a * 9, c = r / 3, b = r - c * 3;
    f = field;
    vs = d.cells();
    ra = a; rb = 3 + b; rc = 6 + c;
    off = ((c - 1) * d.n2 + (b - 1)) * d.n1 + (a - 1);
    on = lane < 27 && (d.three_d || c == 1);
    cur = kNoCell;
    base = 0;
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  }
  __device__ __forceinline__ void add_acc(bool who) {
    if (!who) return;
    double *t = f + base + off;
#pragma unroll
    for (int v = 0; v < NV; ++v)
      if (acc[v] != 0.0) atomicAdd(t + v * vs, acc[v]);
  }
  __device__ __forceinline__ void flush() {
    if (cur != kNoCell) add_acc(on);
    cur = kNoCell;
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  }
  // the window moved to anchor cell k (field index kb)
  __device__ __forceinline__ void move_to(unsigned k, long long kb) {
    if (cur != kNoCell && k == cur + 1) {
      // the next cell of the row (a row's last padded cell is no anchor, so cur + 1 is never
      // the next row's): column 0 is finished, columns 1 and 2 become 0 and 1
      const int lane = threadIdx.x & 31;
      add_acc(on && lane < 9);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const double y = __shfl_down_sync(0xffffffffu, acc[v], 9);
        acc[v] = lane < 18 ? y : 0.0;
      }
    } else {
      flush();
    }
    cur = k;
    base = kb;
  }
  __device__ __forceinline__ void one(const WarpStage &s, int p, bool take) {
    double wcb = s.w[rc][p] * s.w[rb][p];
    const double2 q01 = *(const double2 *)&s.q[p][0];
    const double2 q23 = *(const double2 *)&s.q[p][2];
    if (FAC) wcb *= q01.x;
    if (!take || wcb == 0.0) return;
    const double w = wcb * s.w[ra][p];
    const double val[4] = {q01.x, q01.y, q23.x, q23.y};
    if (ONE) acc[0] += w;
#pragma unroll
    for (int v = ONE ? 1 : 0; v < NV; ++v)
      acc[v] = __fma_rn(w, val[v - (ONE ? 1 : 0) + (FAC ? 1 : 0)], acc[v]);
  }
  // the staged batch: key this lane's anchor cell (the padded cell's index over all blocks),
  // kb its index in the field (variable 0); live: the lane holds a particle that deposits
  __device__ __forceinline__ void batch(const WarpStage &s, unsigned key, long long kb,
                                        bool live) {
    unsigned rem = __ballot_sync(0xffffffffu, live);
    while (rem) {
      const bool mine = (rem >> (threadIdx.x & 31)) & 1u;
      const unsigned k = __reduce_min_sync(0xffffffffu, mine ? key : kNoCell);
      unsigned grp = __ballot_sync(0xffffffffu, mine && key == k);
      rem &= ~grp;
      if (k != cur) move_to(k, __shfl_sync(0xffffffffu, kb, __ffs(grp) - 1));
      while (grp) {
        // two particles at a time: their shared loads fly together
        const int p = __ffs(grp) - 1;
        grp &= grp - 1;
        const int p2 = grp ? __ffs(grp) - 1 : p;
        const bool two = grp != 0;
        grp &= grp - 1;                            // (0 & x stays 0)
        one(s, p, true);
        one(s, p2, two);
      }
    }
  }
};

static_assert(sizeof(WarpStage) % 16 == 0, "the stages of a CTA follow one another");

}  // namespace dustb
