// gpr_multi.cuh - level-set ghost fluid on the device (one level set, at most
// two materials, no heat conduction: the V = 15 layout).
//
// Restates the reference's multi/ module and the interface Riemann problem
// it calls:
//   re-distancing        multi/pfmm.cpp:4-26 (first-order fast marching of
//                        the vendored scikit-fmm, distance_marcher.cpp,
//                        base_marcher.cpp)
//   normals              multi/functions.cpp:16-54 (finite_difference)
//   interface cells      multi/fill.cpp:20-74 (find_interface_cells)
//   boundary fill        multi/fill.cpp:96-235 (fill_boundary_cells)
//   layered fill         multi/fill.cpp:237-328 (fill_neighbor_cells)
//   star state           system/multi/riemann.cpp:26-233, conditions.cpp,
//                        rotations.cpp, functions/vectors.cpp:85-154
//   merge, CFL, renorm   solvers/iterator.cpp:12-83, solvers/utils.cpp:6-23
//
// The reference runs every piece as a sequential sweep over the grid.  Here
// each is a data-parallel kernel whose result equals the sequential sweep:
//   * the fast marching order is replaced by tiled sweeps of the same
//     causal upwind update, whose fixed point is what the marcher computes
//     (band neighbours always enter a point's quadratic, the others only
//     while their distance is below the point's estimate, as the marcher's
//     heap order makes it), in FP64 with the marcher's quadratic and
//     roundings;
//   * a boundary cell reads the right-hand state of the interface from a
//     cell that an earlier cell of the (i, j) sweep may have filled; those
//     reads are resolved to the last earlier writer and solved level by
//     level (almost every cell is on level 0);
//   * within one layer of the extrapolation, a cell copies from a cell of the
//     same layer only if the sweep reached that one first; that chain is
//     followed explicitly.
#pragma once

#include <float.h>

#include "gpr_kernels.cuh"
#include "gpr_ode.cuh"

namespace gpr {
namespace multi {

// Grid of nd = 1 (ny = 1) or 2 dimensions; cell (i, j) is flat index
// i * ny + j, the reference's cell order.
struct Grid {
  int nd, nx, ny;
  long ncell;
  double dx, dy;
};

// Non-contracted FP64 arithmetic where the result feeds a discontinuous
// decision (index truncation, marcher ordering): the same roundings as the
// reference's separate multiplies and adds.
GPR_D double mul(double a, double b) { return __dmul_rn(a, b); }
GPR_D double add(double a, double b) { return __dadd_rn(a, b); }
GPR_D double sub(double a, double b) { return __dsub_rn(a, b); }
GPR_D double dvd(double a, double b) { return __ddiv_rn(a, b); }

// ===========================================================================
// Re-distancing (first-order fast marching, no narrow band, not periodic).

// Frozen band (initalizeFrozen, distance_marcher.cpp:90-151, with the
// reference's edit: the least per-axis crossing distance): cells where phi
// is zero or changes sign across a face, in FP64 with the marcher's
// roundings.  Others start unknown (+inf).  phi[c * ps] is the level set of
// cell c.  fz: bit 0 frozen (band), bit 1 the marcher would take the
// positive root for this cell (phi > DBL_EPSILON), bit 2 the point waits
// for an update (set by the sweeps); par: the neighbours that entered the
// point's update (set by the sweeps).
__global__ void k_fmm_init(const double *__restrict__ phi, long ps, double *__restrict__ d,
                           uint8_t *__restrict__ fz, uint8_t *__restrict__ par, Grid g,
                           int *__restrict__ anyfrozen, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell)
    return;
  int i = g.nd == 1 ? (int)c : (int)(c / g.ny), j = g.nd == 1 ? 0 : (int)(c % g.ny);
  double p = phi[c * ps];
  uint8_t pos = p > DBL_EPSILON ? 2 : 0;
  double x = INFINITY;
  bool frozen = false;
  if (p == 0.0) {
    x = 0.0;
    frozen = true;
  } else {
    double ld[2] = {0.0, 0.0};
    bool borders = false;
    for (int dim = 0; dim < g.nd; dim++) {
      double h = dim == 0 ? g.dx : g.dy;
      for (int dir = -1; dir < 2; dir += 2) {
        int ii = dim == 0 ? i + dir : i, jj = dim == 1 ? j + dir : j;
        if (ii < 0 || ii >= g.nx || jj < 0 || jj >= g.ny)
          continue;
        double pn = phi[((long)ii * g.ny + jj) * ps];
        if (mul(p, pn) < 0.0) {
          borders = true;
          double dd = dvd(mul(h, p), sub(p, pn));
          if (ld[dim] == 0.0 || ld[dim] > dd)
            ld[dim] = dd;
        }
      }
    }
    if (borders) {
      double m = DBL_MAX;
      for (int dim = 0; dim < g.nd; dim++) {
        double t = fabs(ld[dim]);
        if (t > 0.0)
          m = t < m ? t : m;
      }
      x = p < 0.0 ? -m : m;
      frozen = true;
    }
  }
  d[c] = x;
  fz[c] = (frozen ? 1 : 0) | pos;
  // (2D: the flags again in bits 4 and 5, so that a sweep reads one byte)
  par[c] = g.nd == 2 ? ((frozen ? 1 : 0) | pos) << 4 : 0;
  if (frozen)
    atomicOr(anyfrozen, 1);
}

// Grid constants of the update: the marcher's idx2 = 1 / dx^2, 1 / dy^2
// (distance_marcher.cpp), its quadratic's leading coefficient for each set
// of entered axes (idx2[0], idx2[1], idx2[0] + idx2[1], as the marcher sums
// it) and that coefficient's reciprocal rounded to nearest, and the
// spacings.
struct FmmConst {
  double idx2[2], a[3], a4[3], ra[3], h[2], ih[2];
};

inline FmmConst fmm_const(double dx, double dy) {
  FmmConst K;
  K.idx2[0] = 1.0 / dx / dx;
  K.idx2[1] = 1.0 / dy / dy;
  K.a[0] = K.idx2[0];
  K.a[1] = K.idx2[1];
  K.a[2] = K.idx2[0] + K.idx2[1];
  for (int k = 0; k < 3; k++) {
    K.a4[k] = 4.0 * K.a[k];
    K.ra[k] = 1.0 / K.a[k];
  }
  K.h[0] = dx;
  K.h[1] = dy;
  K.ih[0] = 1.0 / dx;
  K.ih[1] = 1.0 / dy;
  return K;
}

// |x| compares as the integer of its bits (the order of |x| for finite
// values and infinity), on the integer pipe.
GPR_D unsigned long long fmm_key(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}

// updatePointOrderOne + solveQuadratic (distance_marcher.cpp:5-28, 72-88)
// for the entered axes (use): a = sum idx2, b = -sum 2 idx2 v, c = sum idx2
// v^2 - 1, root (-b +- sqrt(b^2 - 4ac)) / 2 / a by the sign of phi, in FP64
// with the marcher's operation order and the fused multiply-adds of the
// reference's -O3 -march=native build (CMakeLists.txt:14): b and c
// accumulate by fma, det = fma(b, b, -(4 a c)); every other operation is
// rounded on its own.  The halving is a multiply by 0.5 (exact, the same
// value) and the division by a is Markstein's correction of a product with
// the rounded reciprocal, q = RN(q0 + RN(x - a q0) ra) with q0 = RN(x ra)
// (P. Markstein, IBM J. Res. Dev. 34, 1990; the correctly rounded quotient
// when ra = RN(1/a), as __ddiv_rn gives it).  The marcher leaves a point
// unchanged when the quadratic has no real root (its 0 return); so does a
// false return here.
GPR_D bool fmm_root(const double v[2], const bool use[2], const FmmConst &K, int nd, bool pos,
                    double &x) {
  // a (the sum of the entered idx2, in the marcher's order) and 4a are
  // tabulated per set of entered axes
  double b = 0.0, c = 0.0;
  for (int dim = 0; dim < nd; dim++)
    if (use[dim]) {
      b = __fma_rn(-mul(K.idx2[dim], 2.0), v[dim], b);
      c = __fma_rn(K.idx2[dim], mul(v[dim], v[dim]), c);
    }
  const int ka = use[0] && use[1] ? 2 : (use[0] ? 0 : 1);
  c = sub(c, 1.0);
  const double det = __fma_rn(b, b, -mul(K.a4[ka], c));
  // (comparisons on the bits where they are exact: the integer pipe)
  if (__double_as_longlong(det) <= 0 || fmm_key(det) > 0x7ff0000000000000ull)
    return false;
  const double sq = __dsqrt_rn(det);
  const double num = mul(pos ? add(-b, sq) : sub(-b, sq), 0.5);
  const double q0 = mul(num, K.ra[ka]);
  x = __fma_rn(__fma_rn(-q0, K.a[ka], num), K.ra[ka], q0);
  return fmm_key(x) != 0ull;
}

// Update of one unfrozen point from its neighbours' current values
// (signed; +inf unknown), reproducing what the marcher's heap order makes
// of it (base_marcher.cpp:98-188): band neighbours (frozen at
// initialisation) always enter; the other neighbours enter in increasing
// |d| (equal keys together, as the marcher freezes them in one batch) while
// their |d| is below the point's current estimate, i.e. they were frozen
// before the point; after each entry the quadratic of the entered set is
// the new estimate, or, without a real root, the estimate stays (the
// marcher's 0 return).  Per axis the entered neighbour of least |d| is used
// (the lower one on ties, as the marcher scans -1 then +1).  Where
// rounding makes the new estimate fall below the neighbour that entered (a
// noise-level tie), the marcher keeps it and freezes the point next, so
// the point cannot enter that neighbour: each point records the
// non-band neighbours that entered it (mask bits 2 dim + side), and a
// neighbour that recorded this point is not a candidate here.  Returns
// `old` when nothing is known.
//
// A one-axis root is v +- h up to the quadratic's cancellation (at most
// ~eps (v^2 / h + |v| + h)); it is kept in that form while it only decides
// whether the next neighbour enters and the decision is clear by 256 times
// that bound, and evaluated exactly where it is the result or the decision
// is close.  The result is the same as evaluating every root exactly.
GPR_D double fmm_update(const double nb[2][2], const bool band[2][2], const bool excl[2][2],
                        bool pos, int nd, double old, const FmmConst &K, int &mask) {
  const double INF = INFINITY;
  const unsigned long long KINF = 0x7ff0000000000000ull;
  double v[2] = {INF, INF}, cv[2] = {INF, INF};
  unsigned long long ck[2] = {KINF, KINF};
  int cs[2] = {0, 0};
  bool use[2] = {false, false};
  for (int dim = 0; dim < nd; dim++)
    for (int s = 0; s < 2; s++) {
      const double x = nb[dim][s];
      const unsigned long long kx = fmm_key(x);
      if (band[dim][s]) {
        if (!use[dim] || kx < fmm_key(v[dim])) {
          v[dim] = x;
          use[dim] = true;
        }
      } else if (!excl[dim][s] && kx < ck[dim]) {
        ck[dim] = kx;
        cv[dim] = x;
        cs[dim] = s;
      }
    }
  mask = 0;
  double t = INF, tm = 0.0;  // tm > 0: t is v +- h, within tm of the exact root
  if (use[0] || use[1]) {
    double r;
    if (fmm_root(v, use, K, nd, pos, r))
      t = r;
  }
  bool done[2] = {ck[0] == KINF, nd < 2 || ck[1] == KINF};
  while (!done[0] || !done[1]) {
    const int a = done[0] ? 1 : (done[1] ? 0 : (ck[1] < ck[0] ? 1 : 0));
    const unsigned long long key = ck[a];
    if (tm > 0.0 && fabs(fabs(cv[a]) - fabs(t)) <= tm) {
      double r;
      if (fmm_root(v, use, K, nd, pos, r))
        t = r;
      tm = 0.0;
    }
    if (!(key < fmm_key(t)))
      break;
    const bool both = !done[1 - a] && ck[1 - a] == key;
    for (int q = 0; q < 2; q++) {
      const int dim = q == 0 ? a : 1 - a;
      if (q == 1 && !both)
        break;
      if (!use[dim] || fmm_key(cv[dim]) < fmm_key(v[dim])) {
        v[dim] = cv[dim];
        use[dim] = true;
      }
      mask |= 1 << (2 * dim + cs[dim]);
      done[dim] = true;
    }
    if (use[0] && use[1]) {
      double r;
      if (fmm_root(v, use, K, nd, pos, r)) {
        t = r;
        tm = 0.0;
      }
    } else {
      // v +- h of the one entered axis, and the bound of its distance from
      // the marcher's root
      const int k = use[0] ? 0 : 1;
      const double w = fabs(v[k]), h = K.h[k];
      const double t2 = pos ? v[k] + h : v[k] - h;
      const double m2 = 256.0 * DBL_EPSILON * (w * w * K.ih[k] + w + h);
      if (fabs(t2) > m2) {
        t = t2;
        tm = m2;
      } else {
        double r;
        if (fmm_root(v, use, K, nd, pos, r)) {
          t = r;
          tm = 0.0;
        }
      }
    }
  }
  if (tm > 0.0) {
    double r;
    if (fmm_root(v, use, K, nd, pos, r))
      t = r;
  }
  return isinf(t) ? old : t;
}

// fmm_update in 2D, with one root for all lanes of a warp.  Away from the band
// the entered set is decided from v +- h alone (above), so the smaller
// neighbour enters, the other one enters or not, and the quadratic of the
// final set is evaluated once; in fmm_update the one- and two-axis roots
// are different branches, which a warp takes one after the other.  Band
// neighbours, close decisions and quadratics without a real root take
// fmm_update itself.  The value and the mask are fmm_update's bit for bit.
GPR_D double fmm_update_2d(const double nb[2][2], const bool band[2][2], const bool excl[2][2],
                           bool pos, double old, const FmmConst &K, int &mask) {
  const unsigned long long KINF = 0x7ff0000000000000ull;
  double v[2] = {INFINITY, INFINITY};
  unsigned long long ck[2] = {KINF, KINF};
  int cs[2] = {0, 0};
#pragma unroll
  for (int dim = 0; dim < 2; dim++)
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const unsigned long long kx = fmm_key(nb[dim][s]);
      if (!excl[dim][s] && kx < ck[dim]) {
        ck[dim] = kx;
        v[dim] = nb[dim][s];
        cs[dim] = s;
      }
    }
  const bool second = ck[1] < ck[0], tie = ck[0] == ck[1];
  const double va = second ? v[1] : v[0], h = second ? K.h[1] : K.h[0];
  const double wb = fabs(second ? v[0] : v[1]), t = fabs(va + (pos ? h : -h));
  // the bound in FP32, from high words (relative error below 2^-19, an
  // overflow or NaN makes every comparison false)
  const float wf = f32_abs_hi(va), hf = f32_abs_hi(h) * 1.00001f;
  const float tm = 1.0001f * 256.0f * (float)DBL_EPSILON *
                   (wf * (wf * f32_abs_hi(second ? K.ih[1] : K.ih[0])) + wf + hf);
  const bool both = tie || fmm_key(wb) < fmm_key(t);
  const bool use[2] = {both || !second, both || second};
  bool easy = !(band[0][0] || band[0][1] || band[1][0] || band[1][1]);
  easy = easy && (tie || (f32_abs_hi(t) > tm && f32_abs_hi(wb - t) > tm));
  double x;
  easy = fmm_root(v, use, K, 2, pos, x) && easy && fmm_key(x) < KINF;
  if (!easy)
    return fmm_update(nb, band, excl, pos, 2, old, K, mask);
  mask = (use[0] ? 1 << cs[0] : 0) | (use[1] ? 4 << cs[1] : 0);
  return x;
}

// The four neighbours of shared-memory point m (x neighbours m -+ o0, y
// neighbours m -+ 1) and whether each is in the frozen band.
template <int ND>
GPR_D void fmm_load_nb(const double *src, const uint8_t *sf, int m, int o0, double nb[2][2],
                       bool bd[2][2]) {
  nb[0][0] = src[m - o0];
  nb[0][1] = src[m + o0];
  bd[0][0] = sf[m - o0] & 1;
  bd[0][1] = sf[m + o0] & 1;
  if (ND == 2) {
    nb[1][0] = src[m - 1];
    nb[1][1] = src[m + 1];
    bd[1][0] = sf[m - 1] & 1;
    bd[1][1] = sf[m + 1] & 1;
  } else {
    nb[1][0] = nb[1][1] = INFINITY;
    bd[1][0] = bd[1][1] = false;
  }
}

// One round of tiled Jacobi sweeps of the causal update, in FP64.  Each
// block loads its tile and a one-cell halo into shared memory and runs up
// to `nsweeps` sweeps against that halo, then writes back.  A point waits
// for an update (dirty) when a neighbour changed after its last update;
// each sweep gathers the waiting points into a list first, so that whole
// warps run the updates, and a changed point makes its unfrozen tile
// neighbours wait.  GB300's FP64 pipe issues one warp instruction per 64
// cycles per SM partition, so the sweeps' cost is the longest chain of
// dependent updates (~1400 sweeps at 800 x 400, a tile crossed per round)
// times the update's FP64 instruction count, which the update above keeps
// to about one root.  The sweeps end when no point waits, at the fixed
// point of the update, whatever the order of the work.  lastg[c] is the
// round of cell c's last change; fz bit 2 carries a waiting point into the
// next round.  A tile runs if it has waiting points or a neighbouring tile
// changed in the previous round (tflag bit 1 / bit 0 of round - 1);
// flags[round] records whether anything changed or waits, and a round after
// a round without either returns at once.  2D tiles are 32 x 32 cells, 1D
// tiles 1024.  On the 800 x 400 shock bubble 8 x 8 tiles take the step
// from 23.8 to 22.5 ms against 16 x 16 ones: the front's tiles spread over
// more SMs, though the sweeps make more updates (33 per cell on the static
// circle, 91 after 13 steps of advection, against 34 and 60) along about
// the same chain of 1350-1650 dependent sweeps.  Each thread owns one 2D
// cell or two 1D cells.
constexpr int FMM_T2 = 8, FMM_T1 = 1024;
template <int ND> struct FmmThreads {
  static constexpr int value = ND == 2 ? 64 : 512;
};

template <int ND>
__global__ void __launch_bounds__(FmmThreads<ND>::value, ND == 2 ? 16 : 2)
    k_fmm_round(double *__restrict__ d, uint8_t *__restrict__ fz, uint8_t *__restrict__ par,
                int *__restrict__ lastg, Grid g, FmmConst K, int *__restrict__ flags, int *__restrict__ tflag, int round,
                int nsweeps, int mono, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  if (round > 0 && flags[round - 1] == 0)
    return;
  constexpr int TX = ND == 2 ? FMM_T2 : FMM_T1, TY = ND == 2 ? FMM_T2 : 1;
  constexpr int SX = TX + 2, SY = ND == 2 ? TY + 2 : 1;
  constexpr int FMM_THREADS = FmmThreads<ND>::value;
  constexpr int NT = TX * TY, PER = NT / FMM_THREADS, NW = FMM_THREADS / 32;
  const int ntx0 = (g.nx + TX - 1) / TX, nty0 = ND == 2 ? (g.ny + TY - 1) / TY : 1;
  const int ntiles = ntx0 * nty0;
  const int t = blockIdx.x;
  if (round > 0) {
    const int *prev = tflag + (long)(round - 1) * ntiles;
    int ti = ND == 2 ? t % ntx0 : t, tj = ND == 2 ? t / ntx0 : 0;
    bool run = prev[t] != 0 || (ti > 0 && (prev[t - 1] & 1)) ||
               (ti < ntx0 - 1 && (prev[t + 1] & 1)) ||
               (ND == 2 && ((tj > 0 && (prev[t - ntx0] & 1)) ||
                            (tj < nty0 - 1 && (prev[t + ntx0] & 1))));
    if (!run)
      return;
  }
  __shared__ double sd[SX * SY];
  __shared__ double nvs[NT];
  __shared__ uint8_t sf[SX * SY];
  __shared__ uint8_t sp[SX * SY];    // the neighbours that entered each point
  __shared__ uint8_t nms[NT];        // new masks of a sweep's updates
  __shared__ uint8_t hchg[SX * SY];  // halo point changed in the previous round
  __shared__ uint8_t dirty[NT];
  __shared__ uint8_t chg[NT];  // changed in this round
  __shared__ int16_t list[NT];
  __shared__ int wcnt[NW], total;
  const int bi = ND == 2 ? t % ntx0 : t, bj = ND == 2 ? t / ntx0 : 0;
  const int i0 = bi * TX, j0 = bj * TY;
  for (int e = threadIdx.x; e < SX * SY; e += FMM_THREADS) {
    int a = ND == 2 ? e / SY : e, b = ND == 2 ? e % SY : 0;
    int ii = i0 + a - 1, jj = ND == 2 ? j0 + b - 1 : 0;
    double x = INFINITY;
    uint8_t f = 0, hc = 0, pm = 0;
    if (ii >= 0 && ii < g.nx && jj >= 0 && jj < g.ny) {
      long c = (long)ii * g.ny + jj;
      x = d[c];
      f = fz[c];
      pm = par[c];
      hc = lastg[c] == round - 1;
    }
    sd[e] = x;
    sf[e] = f;
    sp[e] = pm;
    hchg[e] = hc;
  }
  auto smem_of = [&](int l) {
    return ND == 2 ? (l / TY + 1) * SY + (l % TY + 1) : l + 1;
  };
  auto inside_of = [&](int l) {
    int i = i0 + (ND == 2 ? l / TY : l), j = ND == 2 ? j0 + l % TY : 0;
    return i < g.nx && j < g.ny;
  };
  auto cell_of = [&](int l) {
    int i = i0 + (ND == 2 ? l / TY : l), j = ND == 2 ? j0 + l % TY : 0;
    return (long)i * g.ny + j;
  };
  auto is_halo = [&](int m) {
    int a = ND == 2 ? m / SY : m, b = ND == 2 ? m % SY : 1;
    return a == 0 || a == SX - 1 || (ND == 2 && (b == 0 || b == SY - 1));
  };
  const int o0 = ND == 2 ? SY : 1;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  bool act[PER];
  for (int k = 0; k < PER; k++) {
    const int l = threadIdx.x + k * FMM_THREADS, m = smem_of(l);
    act[k] = inside_of(l) && !(sf[m] & 1);
    bool dd = act[k] && (round == 0 || (sf[m] & 4));
    if (act[k] && !dd) {
      const int nbm[4] = {m - o0, m + o0, m - 1, m + 1};
      for (int q = 0; q < (ND == 2 ? 4 : 2); q++)
        dd = dd || (is_halo(nbm[q]) && hchg[nbm[q]]);
    }
    dirty[l] = dd;
    chg[l] = 0;
  }
  __syncthreads();
  for (int it = 0; it < nsweeps; it++) {
    // 1. gather the waiting points (each thread clears its own flags)
    int mine = 0;
    bool sel[PER];
    for (int k = 0; k < PER; k++) {
      const int l = threadIdx.x + k * FMM_THREADS;
      sel[k] = dirty[l] != 0;
      dirty[l] = 0;
      mine += sel[k];
    }
    int incl = mine;  // inclusive warp scan
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o)
        incl += y;
    }
    if (lane == 31)
      wcnt[wid] = incl;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < wid; w++)
      base += wcnt[w];
    int pos = base + incl - mine;
    for (int k = 0; k < PER; k++)
      if (sel[k])
        list[pos++] = (int16_t)(threadIdx.x + k * FMM_THREADS);
    if (threadIdx.x == FMM_THREADS - 1)
      total = pos;
    __syncthreads();
    const int n = total;
    if (n == 0)
      break;
    // 2. updates (Jacobi: read the neighbours, write after a barrier)
    for (int q = threadIdx.x; q < n; q += FMM_THREADS) {
      const int m = smem_of(list[q]);
      double nb[2][2];
      bool bd[2][2];
      fmm_load_nb<ND>(sd, sf, m, o0, nb, bd);
      // a neighbour that recorded this point as entered (its bit for the
      // opposite side) is not a candidate
      bool ex[2][2];
      ex[0][0] = (sp[m - o0] >> 1) & 1;
      ex[0][1] = sp[m + o0] & 1;
      ex[1][0] = ND == 2 && ((sp[m - 1] >> 3) & 1);
      ex[1][1] = ND == 2 && ((sp[m + 1] >> 2) & 1);
      int msk;
      nvs[q] = fmm_update(nb, bd, ex, (sf[m] & 2) != 0, ND, sd[m], K, msk);
      nms[q] = (uint8_t)msk;
    }
    __syncthreads();
    // 3. take the new values (from the second half of the round budget on,
    // only a smaller |d|, which guarantees termination); the unfrozen tile
    // neighbours of a changed point wait for the next sweep
    for (int q = threadIdx.x; q < n; q += FMM_THREADS) {
      const int l = list[q], m = smem_of(l);
      const double old = sd[m], nv = nvs[q];
      if (mono ? fabs(nv) < fabs(old) : (nv != old || nms[q] != sp[m])) {
        sd[m] = nv;
        sp[m] = nms[q];
        chg[l] = 1;
        const int nbm[4] = {m - o0, m + o0, m - 1, m + 1};
        const int nbl[4] = {ND == 2 ? l - TY : l - 1, ND == 2 ? l + TY : l + 1, l - 1, l + 1};
        for (int k = 0; k < (ND == 2 ? 4 : 2); k++)
          if (!is_halo(nbm[k]) && !(sf[nbm[k]] & 1) && inside_of(nbl[k]))
            dirty[nbl[k]] = 1;
      }
    }
    __syncthreads();
  }
  bool wrote = false, waits = false;
  for (int k = 0; k < PER; k++) {
    const int l = threadIdx.x + k * FMM_THREADS;
    if (!act[k])
      continue;
    const int m = smem_of(l);
    const long c = cell_of(l);
    if (chg[l]) {
      d[c] = sd[m];
      par[c] = sp[m];
      lastg[c] = round;
      wrote = true;
    }
    const uint8_t f = (sf[m] & 3) | (dirty[l] ? 4 : 0);
    if (f != sf[m])
      fz[c] = f;
    waits = waits || dirty[l];
  }
  const bool any_wrote = __syncthreads_or(wrote);
  const bool any_waits = __syncthreads_or(waits);
  if (threadIdx.x == 0) {
    const int fl = (any_wrote ? 1 : 0) | (any_waits ? 2 : 0);
    tflag[(long)round * ntiles + t] = fl;
    if (fl)
      atomicOr(&flags[round], 1);
  }
}

// ---------------------------------------------------------------------------
// 2D re-distancing as one persistent grid: global Jacobi sweeps of the same
// update (fmm_update), one grid barrier per sweep.  The tiled rounds above
// exchange halos only between launches, so information crosses a tile per
// round and each tile re-sweeps its points until its halo settles (33-91
// updates per cell on the 800 x 400 bubble).  Here every sweep sees the
// previous sweep's values everywhere: a sweep updates only the points that
// changed, or whose neighbours changed, in the previous sweep, the front
// moves a cell per sweep, and the number of sweeps is the depth of the
// marcher's dependency chain (~1.3 x the largest distance in cells: 680
// sweeps of 14400 points, a ring ~25 cells wide, on that bubble).
//
// What bounds it is a sweep's latency, not its work (3 warps of points per
// SM): the waiting points are marked in a byte map, a plain store that
// nobody waits for; each block reads the map of its own cells (dealt out in
// segments of 8, so that a front's ring falls on all SMs alike) in passes of
// 4096 cells, two passes' words in flight beside the one it works on, gathers
// the marked ones into a list in shared memory and, when all passes are read or
// the list could not take another, updates them, a lane each; then the
// barrier.  On the evolved 800 x 400 bubble, one pass, a sweep of 13000 cycles
// (6.7 us) spends 2500 on the map and the list, 5000 on the update (43 FP64
// instructions at 64 cycles a warp) and 5500 on the barrier, whose release
// waits for the sweep's stores.
//
// Lists of points in global memory with a stamp per point, the other form, cost
// 5500 cycles a sweep for the dependent atomics that dedupe and append, but read
// no cell that does not wait.  Microseconds a sweep, this form and that: a circle
// on 800 x 400 5.3 and 11.0, 1600 x 800 10.1 and 19.0, 3200 x 1600 28 and 50,
// 4096^2 118 and 212; a front along a strip, where the fewest points wait for
// the cells, 64 x 65536 9.8 and 11.3, 512 x 8192 15.9 and 19.7.  An update in
// each pass would cost 22 and 31 on those two.  Also measured at 800 x 400:
// stamping only the changed point and reading the map around each segment,
// fewer stores and seven loads for one (8.2 us); whole parts of the grid in
// shared memory, exchanging frames every 4 sweeps, where the ring falls on few
// of them (25 us).
//
// Jacobi with two buffers: sweep s reads d[s % 2] / par[s % 2] and writes
// d[(s + 1) % 2] / par[(s + 1) % 2] for its marked points; a point that
// changes marks itself for the next sweep as well as its neighbours, which
// copies its new value into the other buffer, so after sweep s the written
// buffer holds every point's latest value.  The fixed point, and so the
// result, is that of the tiled form: the sweeps end when no point changes,
// whatever the order of the work.  From sweep mono_from on only smaller |d|
// is taken (termination, as the tiled form's last rounds); a change still
// found in sweep max_sweeps - 1 sets err bit 0.
//
// The blocks wait for one another at the barrier, so the kernel is launched
// cooperatively (all blocks resident); each wait is bounded (~1 s), after
// which the block sets err bit 2 and leaves.
struct FmmGlobal {
  double *d[2];
  uint8_t *par[2];
  const uint8_t *fz;
  uint8_t *map[2];          // a byte per cell: waits for sweep s (map[s % 2])
  unsigned long long *bar;  // the barrier's two words
  int *err;
  int *sweeps;  // optional: receives the sweeps taken
  int mono_from, max_sweeps;
};

// GPU-scope release / acquire accesses (PTX memory model, sm_70 and later).
GPR_D void fmm_add_release64(unsigned long long *p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" : : "l"(p), "l"(v) : "memory");
}
GPR_D unsigned long long fmm_ld_acquire(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier at the end of sweep s, which also sums what the blocks report
// (changed: 1 if any of the block's points did): the 64-bit word words[s % 2]
// counts the arrivals (bits 40..63) and the reports (bits 0..39) over the
// sweeps of that parity.  Each block arrives once (one thread, a release add
// after the block barrier, which orders the block's writes before it) and
// waits with acquire loads until all blocks have arrived for this sweep:
// nblocks (s / 2 + 1) arrivals.  Two words, so that a block already at the
// next sweep's barrier cannot be counted here.  The sweep's sum is the
// word's growth since the previous sweep of the same parity (prev[2], kept
// by the block).  The wait gives up after ~1 s (err bit 2).  Returns the
// sum, or -1 after a timeout.
GPR_D int fmm_grid_sync(unsigned long long *words, unsigned nblocks, int s, int changed,
                        unsigned long long prev[2], int *err) {
  __shared__ int shn;
  constexpr unsigned long long ARR = 1ull << 40, CNT = ARR - 1;
  // the block barrier is the caller's (it also makes `changed`)
  if (threadIdx.x == 0) {
    const int k = s & 1;
    unsigned long long *w = words + k;
    const unsigned long long target = (unsigned long long)nblocks * (unsigned)(s / 2 + 1);
    fmm_add_release64(w, ARR + (unsigned)changed);
    unsigned long long v = fmm_ld_acquire(w);
    const long long t0 = clock64();
    int n = 0;
    while ((v >> 40) < target) {
      if (clock64() - t0 > 2000000000LL) {  // ~1 s at 2 GHz
        atomicOr(err, 4);
        n = -1;
        break;
      }
      v = fmm_ld_acquire(w);
    }
    if (n == 0) {
      n = (int)((v & CNT) - (k ? prev[1] : prev[0]));
      (k ? prev[1] : prev[0]) = v & CNT;
    }
    shn = n;
  }
  __syncthreads();
  return shn;
}

// The first map: unfrozen points next to the frozen band.
__global__ void k_fmm_seed(Grid g, FmmGlobal G, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  const long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell || (G.fz[c] & 1))
    return;
  const int i = c / g.ny, j = c % g.ny;
  if ((i > 0 && (G.fz[c - g.ny] & 1)) || (i < g.nx - 1 && (G.fz[c + g.ny] & 1)) ||
      (j > 0 && (G.fz[c - 1] & 1)) || (j < g.ny - 1 && (G.fz[c + 1] & 1)))
    G.map[0][c] = 1;
}

constexpr int FMM_G_THREADS = 256, FMM_G_SEGS = 2;  // segments per thread and pass
constexpr int FMM_G_PASS = FMM_G_THREADS * FMM_G_SEGS * 8;  // cells a pass may list

__global__ void __launch_bounds__(FMM_G_THREADS) k_fmm_global(Grid g, FmmConst K, FmmGlobal G,
                                                              const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  constexpr int NT = FMM_G_THREADS, U = FMM_G_SEGS;
  __shared__ int list[2 * FMM_G_PASS], nlist;
  const int tid = threadIdx.x, lane = tid & 31, nb = gridDim.x;
  const int nseg = (int)((g.ncell + 7) / 8), ngroup = (nseg + nb - 1) / nb;
  // Segment of this block in group k of nb consecutive ones: the blocks take
  // them in turn, shifted by 61 from group to group (152 = 8 x 19), since a
  // grid whose rows are whole groups would give a column to one block.  A
  // thread's groups lie NT * U apart, so its place in them moves by `hop`.
  const int hop = (int)((61L * NT * U) % nb);
  int place0[U];
#pragma unroll
  for (int u = 0; u < U; u++)
    place0[u] = ((int)blockIdx.x + nb - (int)((61L * (u * NT + tid)) % nb)) % nb;
  if (tid == 0)
    nlist = 0;
  __syncthreads();
  unsigned long long prev[2] = {0ull, 0ull};  // used by thread 0
  int s = 0, n = 1;
  for (; s < G.max_sweeps && n > 0; s++) {
    const double *src = G.d[s & 1];
    double *dst = G.d[(s + 1) & 1];
    const uint8_t *psrc = G.par[s & 1];
    uint8_t *pdst = G.par[(s + 1) & 1];
    uint8_t *map = G.map[s & 1], *next = G.map[(s + 1) & 1];
    const bool mono = s >= G.mono_from;
    bool any = false;
    // the words of this pass and the next two (loads in flight meanwhile)
    uint2 w[3][U];
    int seg[3][U], place[U];
    auto fetch = [&](int slot, int k0) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int k = k0 + u * NT + tid;
        seg[slot][u] = k * nb + place[u];
        // (the map's last segment ends within its padding)
        w[slot][u] = k < ngroup && seg[slot][u] < nseg
                         ? __ldcg((const uint2 *)map + seg[slot][u])
                         : make_uint2(0u, 0u);
        place[u] -= hop;
        place[u] += place[u] < 0 ? nb : 0;
      }
    };
#pragma unroll
    for (int u = 0; u < U; u++)
      place[u] = place0[u];
    fetch(0, 0);
    if (NT * U < ngroup)
      fetch(1, NT * U);
    for (int k0 = 0; k0 < ngroup; k0 += NT * U) {
      const bool more = k0 + NT * U < ngroup;
      if (k0 + 2 * NT * U < ngroup)
        fetch(2, k0 + 2 * NT * U);
      unsigned bits = 0;  // 8 u + b: cell b of segment u
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (w[0][u].x | w[0][u].y)
          __stcg((uint2 *)map + seg[0][u], make_uint2(0u, 0u));
        // bytes 0 or 1, the four bytes' bits together
        const unsigned lo = w[0][u].x, hi = w[0][u].y;
        bits |= (((lo * 0x01020408u) >> 24) | ((hi * 0x01020408u) >> 24) << 4) << (8 * u);
      }
      int end = 0;  // entries listed so far, as this warp knows
      if (__any_sync(0xffffffffu, bits != 0u)) {
        int incl = __popc(bits);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          incl += lane >= o ? y : 0;
        }
        int pos = 0;
        if (lane == 31)
          pos = atomicAdd(&nlist, incl);
        pos = __shfl_sync(0xffffffffu, pos, 31) + incl;
        end = pos;
        pos -= __popc(bits);
        while (bits) {
          const int b = __ffs(bits) - 1;
          bits &= bits - 1;
          int sg = seg[0][0];
#pragma unroll
          for (int u = 1; u < U; u++)
            sg = (b >> 3) == u ? seg[0][u] : sg;
          list[pos++] = sg * 8 + (b & 7);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        w[0][u] = w[1][u];
        seg[0][u] = seg[1][u];
        w[1][u] = w[2][u];
        seg[1][u] = seg[2][u];
      }
      // updates wait until the list could not take another pass
      if (more && !__syncthreads_or(end > FMM_G_PASS))
        continue;
      __syncthreads();
      const int nl = nlist;
      for (int q = tid; q < nl; q += NT) {
        const int c = list[q];
        const int i = c / g.ny, j = c - i * g.ny;
        double nb4[2][2];
        bool bd[2][2], ex[2][2];
        const int cn[2][2] = {{c - g.ny, c + g.ny}, {c - 1, c + 1}};
        const bool in[2][2] = {{i > 0, i < g.nx - 1}, {j > 0, j < g.ny - 1}};
        // a neighbour that recorded this point as entered (its bit for the
        // opposite side) is not a candidate: bits 2 dim + side
        const int xb[2][2] = {{1, 0}, {3, 2}};
#pragma unroll
        for (int dim = 0; dim < 2; dim++)
#pragma unroll
          for (int sd = 0; sd < 2; sd++) {
            const bool ok = in[dim][sd];
            const int m = ok ? cn[dim][sd] : c;
            const double x = __ldcg(src + m);
            const uint8_t pm = __ldcg(psrc + m);
            nb4[dim][sd] = ok ? x : INFINITY;
            bd[dim][sd] = ok && (pm & 16);
            ex[dim][sd] = ok && ((pm >> xb[dim][sd]) & 1);
          }
        const double old = __ldcg(src + c);
        const uint8_t pold = __ldcg(psrc + c);
        int msk;
        const double nv = fmm_update_2d(nb4, bd, ex, (pold & 32) != 0, old, K, msk);
        const bool chg = mono ? fmm_key(nv) < fmm_key(old)
                              : (__double_as_longlong(nv) != __double_as_longlong(old) ||
                                 msk != (pold & 15));
        __stcg(dst + c, chg ? nv : old);
        __stcg(pdst + c, chg ? (uint8_t)(msk | (pold & 48)) : pold);
        if (chg) {  // the point itself and its neighbours wait for sweep s + 1
          any = true;
          __stcg(next + c, (uint8_t)1);
#pragma unroll
          for (int dim = 0; dim < 2; dim++)
#pragma unroll
            for (int sd = 0; sd < 2; sd++)
              if (in[dim][sd] && !bd[dim][sd])  // (frozen ones never)
                __stcg(next + cn[dim][sd], (uint8_t)1);
        }
      }
      if (more) {  // the list again, for the next passes
        __syncthreads();
        if (tid == 0)
          nlist = 0;
        __syncthreads();
      }
    }
    const int changed = __syncthreads_or(any);
    if (tid == 0)
      nlist = 0;
    n = fmm_grid_sync(G.bar, (unsigned)nb, s, changed ? 1 : 0, prev, G.err);
    if (n < 0)
      return;
  }
  if (blockIdx.x == 0 && tid == 0) {
    if (n != 0)
      atomicOr(G.err, 1);  // not converged within the sweep budget
    if (G.sweeps)
      *G.sweeps = s;
  }
}

// Final values (base_marcher.cpp:103-106, 190-196): zeros when nothing
// froze, DBL_MAX where the march never arrived; the distance also replaces
// the level set in u (renormalize_levelsets, multi/functions.cpp:56-64).
template <int V>
__global__ void k_fmm_finish(double *__restrict__ d, double *__restrict__ u, long ncell,
                             const int *__restrict__ anyfrozen, const int *__restrict__ flags,
                             int last, int *__restrict__ err, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c == 0 && flags[last] != 0)
    atomicOr(err, 1);  // not converged within the round budget
  if (c >= ncell)
    return;
  double x = d[c];
  if (isinf(x))
    x = DBL_MAX;
  if (!*anyfrozen)
    x = 0.0;
  d[c] = x;
  if (u)
    u[c * V + V - 1] = x;
}

// ===========================================================================
// Normals and interface cells of one material from its level set phi
// (material_indicator, multi/functions.cpp:66-81: phi = +-u's level set for
// two materials; the material occupies phi <= 0).

__global__ void k_mat_phi(const double *__restrict__ d, int sgn, double *__restrict__ phim,
                          long ncell, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c < ncell)
    phim[c] = sgn > 0 ? d[c] : -d[c];
}

// finite_difference (multi/functions.cpp:16-54): central differences, the
// first and last rows (columns) copied from their neighbours.  dphi is
// [ncell][nd].
__global__ void k_finite_difference(const double *__restrict__ phi, double *__restrict__ dphi,
                                    Grid g, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell)
    return;
  if (g.nd == 1) {
    int i = (int)c, ii = i == 0 ? 1 : (i == g.nx - 1 ? g.nx - 2 : i);
    dphi[c] = dvd(sub(phi[ii + 1], phi[ii - 1]), mul(2.0, g.dx));
    return;
  }
  int i = (int)(c / g.ny), j = (int)(c % g.ny);
  int ii = i == 0 ? 1 : (i == g.nx - 1 ? g.nx - 2 : i);
  int jj = j == 0 ? 1 : (j == g.ny - 1 ? g.ny - 2 : j);
  dphi[2 * c] = dvd(sub(phi[(long)(ii + 1) * g.ny + j], phi[(long)(ii - 1) * g.ny + j]),
                    mul(2.0, g.dx));
  dphi[2 * c + 1] = dvd(sub(phi[(long)i * g.ny + jj + 1], phi[(long)i * g.ny + jj - 1]),
                        mul(2.0, g.dy));
}

// find_interface_cells (multi/fill.cpp:20-74), gathered per cell: the
// reference's scatter only ever writes sign(phi) of the written cell, or -2
// for an isolated phi <= 0 cell, so each cell's final value follows from its
// own neighbourhood.
GPR_D bool nonisolated(const double *phi, int i, int j, const Grid &g) {
  long c = (long)i * g.ny + j;
  return (i > 0 && phi[c - g.ny] <= 0.0) || (i < g.nx - 1 && phi[c + g.ny] <= 0.0) ||
         (j > 0 && phi[c - 1] <= 0.0) || (j < g.ny - 1 && phi[c + 1] <= 0.0);
}

__global__ void k_interface_cells(const double *__restrict__ phi, int32_t *__restrict__ im,
                                  Grid g, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell)
    return;
  double p = phi[c];
  int sg = p <= 0.0 ? -1 : 1;
  if (g.nd == 1) {
    int i = (int)c;
    bool hit = (i > 0 && mul(phi[c - 1], p) <= 0.0) ||
               (i < g.nx - 1 && mul(p, phi[c + 1]) <= 0.0);
    im[c] = hit ? sg : 0;
    return;
  }
  int i = (int)(c / g.ny), j = (int)(c % g.ny);
  long nbr[4] = {i > 0 ? c - g.ny : -1, i < g.nx - 1 ? c + g.ny : -1, j > 0 ? c - 1 : -1,
                 j < g.ny - 1 ? c + 1 : -1};
  int ni[4] = {i - 1, i + 1, i, i}, nj[4] = {j, j, j - 1, j + 1};
  int out = 0;
  if (p <= 0.0) {
    if (!nonisolated(phi, i, j, g)) {
      im[c] = -2;
      return;
    }
    for (int q = 0; q < 4; q++)
      if (nbr[q] >= 0 && mul(p, phi[nbr[q]]) <= 0.0)
        out = -1;
  }
  // written by a non-isolated phi <= 0 neighbour whose product with us is <= 0
  for (int q = 0; q < 4 && out == 0; q++) {
    if (nbr[q] < 0)
      continue;
    double pn = phi[nbr[q]];
    if (pn <= 0.0 && mul(pn, p) <= 0.0 && nonisolated(phi, ni[q], nj[q], g))
      out = sg;
  }
  im[c] = out;
}

// ===========================================================================
// Interface Riemann problem (slip conditions, no heat conduction).

// rotation_matrix (rotations.cpp:5-35): rows e1 = n, e2, e3.
GPR_D void rotation(const double n[2], int nd, double R[3][3]) {
  double e1[3] = {n[0], nd == 2 ? n[1] : 0.0, 0.0}, e2[3], e3[3], den;
  double Sq = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
  if (fabs(e1[1] + e1[2]) <= fabs(e1[1] - e1[2])) {
    den = sqrt(2.0 * (1.0 - e1[0] * e1[1] - e1[1] * e1[2] - e1[2] * e1[0]));
    e2[0] = e1[1] - e1[2];
    e2[1] = e1[2] - e1[0];
    e2[2] = e1[0] - e1[1];
    double Sum = e1[0] + e1[1] + e1[2];
    for (int i = 0; i < 3; i++)
      e3[i] = e1[i] * Sum - Sq;
  } else {
    den = sqrt(2.0 * (1.0 + e1[0] * e1[1] + e1[1] * e1[2] - e1[2] * e1[0]));
    e2[0] = e1[1] + e1[2];
    e2[1] = e1[2] - e1[0];
    e2[2] = -e1[0] - e1[1];
    double Sum = e1[0] - e1[1] + e1[2];
    e3[0] = e1[0] * Sum - Sq;
    e3[1] = e1[1] * Sum + Sq;
    e3[2] = e1[2] * Sum - Sq;
  }
  for (int i = 0; i < 3; i++) {
    R[0][i] = e1[i];
    R[1][i] = e2[i] / den;
    R[2][i] = e3[i] / den;
  }
}

// rotate_tensors (rotations.cpp:37-47): v <- R v, A <- R A R^T.
GPR_D void rotate(double *Q, const double R[3][3]) {
  double v[3], T[9];
  for (int i = 0; i < 3; i++)
    v[i] = R[i][0] * Q[2] + R[i][1] * Q[3] + R[i][2] * Q[4];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      T[3 * i + j] = R[i][0] * Q[5 + j] + R[i][1] * Q[8 + j] + R[i][2] * Q[11 + j];
  for (int i = 0; i < 3; i++) {
    Q[2 + i] = v[i];
    for (int j = 0; j < 3; j++)
      Q[5 + 3 * i + j] = T[3 * i] * R[j][0] + T[3 * i + 1] * R[j][1] + T[3 * i + 2] * R[j][2];
  }
}

// Gaussian elimination with partial pivoting: A X = B in place (A n x n,
// B n x m, row-major).  Returns false on a zero pivot.  Rows are exchanged
// one comparison at a time, so that every index is a constant (arrays in
// registers), and each pivot is inverted once.
template <int n, int m> GPR_D bool gauss(double *A, double *B) {
  double ip[n];
#pragma unroll
  for (int c = 0; c < n; c++) {
#pragma unroll
    for (int r = c + 1; r < n; r++) {
      const bool sw = fp_abs_bits(A[r * n + c]) > fp_abs_bits(A[c * n + c]);
#pragma unroll
      for (int j = c; j < n; j++) {
        const double t = A[c * n + j], u = A[r * n + j];
        A[c * n + j] = sw ? u : t;
        A[r * n + j] = sw ? t : u;
      }
#pragma unroll
      for (int j = 0; j < m; j++) {
        const double t = B[c * m + j], u = B[r * m + j];
        B[c * m + j] = sw ? u : t;
        B[r * m + j] = sw ? t : u;
      }
    }
    if (A[c * n + c] == 0.0)
      return false;
    ip[c] = rcp64(A[c * n + c]);
#pragma unroll
    for (int r = c + 1; r < n; r++) {
      const double f = -A[r * n + c] * ip[c];
#pragma unroll
      for (int j = c + 1; j < n; j++)
        A[r * n + j] = fma(f, A[c * n + j], A[r * n + j]);
#pragma unroll
      for (int j = 0; j < m; j++)
        B[r * m + j] = fma(f, B[c * m + j], B[r * m + j]);
    }
  }
#pragma unroll
  for (int c = n - 1; c >= 0; c--)
#pragma unroll
    for (int j = 0; j < m; j++) {
      double t = B[c * m + j];
#pragma unroll
      for (int k = c + 1; k < n; k++)
        t = fma(-A[c * n + k], B[k * m + j], t);
      B[c * m + j] = t * ip[c];
    }
  return true;
}

// Eigenvalues of a real 3 x 3 matrix from its characteristic polynomial
// (depressed cubic: trigonometric form for three real roots, Cardano for a
// complex pair).  ok = false when an eigenvalue has a non-positive real part
// or the pair's imaginary part exceeds 1e-6 of the spectral radius: the
// reference's Q diag(Re(lambda)^(-1/2)) Q^(-1) with Q = Re(eigenvectors)
// (riemann.cpp:136-141) is NaN or singular there and its star state falls
// back to the input state.
static __device__ __noinline__ bool eig3_real_positive(const double *M) {
  double p1 = M[0] + M[4] + M[8];
  double p2 = M[0] * M[4] - M[1] * M[3] + M[0] * M[8] - M[2] * M[6] + M[4] * M[8] -
              M[5] * M[7];
  double p3 = M[0] * (M[4] * M[8] - M[5] * M[7]) - M[1] * (M[3] * M[8] - M[5] * M[6]) +
              M[2] * (M[3] * M[7] - M[4] * M[6]);
  double s = p1 / 3.0;
  double a = p2 - p1 * p1 / 3.0;
  double b = -2.0 * p1 * p1 * p1 / 27.0 + p1 * p2 / 3.0 - p3;
  double disc = b * b / 4.0 + a * a * a / 27.0;  // > 0: complex pair
  if (disc > 0.0) {
    double sq = sqrt(disc);
    double u = cbrt(-b / 2.0 + sq), v = cbrt(-b / 2.0 - sq);
    double lr = s + u + v;                  // real root
    double cr = s - (u + v) / 2.0;          // real part of the pair
    double ci = 0.86602540378443864676 * fabs(u - v);
    double rad = fmax(fabs(lr), hypot(cr, ci));
    return lr > 0.0 && cr > 0.0 && !(ci > 1e-6 * rad);
  }
  // three real roots: s + 2 sqrt(-a/3) cos(theta/3 - 2 pi k / 3)
  double r = sqrt(fmax(-a / 3.0, 0.0));
  double lo;
  if (r == 0.0) {
    lo = s;
  } else {
    double ct = -b / (2.0 * r * r * r);
    ct = fmin(1.0, fmax(-1.0, ct));
    double th = acos(ct);
    // the smallest of the three is k = 1 (theta / 3 + 2 pi / 3 in [2pi/3, pi])
    lo = s + 2.0 * r * cos(th / 3.0 + 2.0943951023931954923);
  }
  return lo > 0.0;
}

// Whether the eigenvalues of M are real and positive, as eig3_real_positive
// decides.  With disc <= 0 the roots are real, and positive exactly when the
// coefficients p1, p2 and p3 are; a complex pair's imaginary part is at most
// sqrt(3 disc) / -a, which settles the rounding-level pairs of a nearly
// isotropic state; anything else takes eig3_real_positive (roots and
// angles).
GPR_D bool spectrum_positive(const double *M) {
  const double m1 = M[4] * M[8] - M[5] * M[7], m2 = M[0] * M[8] - M[2] * M[6],
               m3 = M[0] * M[4] - M[1] * M[3];
  const double p1 = M[0] + M[4] + M[8], p2 = m1 + m2 + m3;
  const double p3 = M[0] * m1 - M[1] * (M[3] * M[8] - M[5] * M[6]) +
                    M[2] * (M[3] * M[7] - M[4] * M[6]);
  const double a = p2 - p1 * p1 * (1.0 / 3.0);
  const double b = p1 * fma(-2.0 / 27.0 * p1, p1, p2 * (1.0 / 3.0)) - p3;
  const double disc = fma(b * b, 0.25, a * a * a * (1.0 / 27.0));
  const double lim = 0.9e-6 / 3.0 * p1 * a;
  bool ok = p1 > 0.0 && p2 > 0.0 && p3 > 1e-10 * p1 * p1 * p1;
  ok = ok && (disc <= 0.0 || (a < 0.0 && 3.0 * disc < lim * lim));
  return ok || eig3_real_positive(M);
}

GPR_D bool inv3(const double *M, double *out) {
  double A[9];
  for (int k = 0; k < 9; k++) {
    A[k] = M[k];
    out[k] = (k % 4) == 0 ? 1.0 : 0.0;
  }
  return gauss<3, 3>(A, out);
}

// Inverse principal square root of a matrix with positive eigenvalues by the
// Denman-Beavers iteration (Y -> M^(1/2), Z -> M^(-1/2)), on M over the mean
// of its eigenvalues; the reference forms the same matrix function from an
// eigen-decomposition (riemann.cpp:136-141).  An update below 3e-9 leaves an
// error of about its square, times the root of the eigenvalues' ratio, so the
// iteration ends with it: 5 iterations for eigenvalues 1 : 1 : 3 (9 unscaled
// and run to a standstill), with the same errors against 64-bit mantissas on
// ratios from 3 (mean 2e-16) to 1e8.  The closed form by the theorem of Cayley
// and Hamilton takes an eighth of the operations and loses a digit.
GPR_D bool inv_sqrt3(const double *M, double *Zout) {
  double Y[9], Z[9], Yi[9], Zi[9];
  const double sc = 3.0 * rcp64(M[0] + M[4] + M[8]);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    Y[k] = M[k] * sc;
    Z[k] = Zi[k] = (k % 4) == 0 ? 1.0 : 0.0;
  }
#pragma unroll 1
  for (int it = 0; it < 100; it++) {
    if (!inv3(Y, Yi) || (it > 0 && !inv3(Z, Zi)))
      return false;
    float dmax = 0.0f, ymax = 0.0f;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double e = 0.5 * (Zi[k] - Y[k]);
      Y[k] += e;
      Z[k] = 0.5 * (Z[k] + Yi[k]);
      dmax = fmaxf(dmax, f32_abs_hi(e));
      ymax = fmaxf(ymax, f32_abs_hi(Y[k]));
    }
    if (!(dmax > 3e-9f * ymax))
      break;
  }
  const double f = sqrt64(sc);
#pragma unroll
  for (int k = 0; k < 9; k++)
    Zout[k] = Z[k] * f;
  return true;
}

// Total stress column 0: Sigma = p e0 - sigma(:, 0)  (variables/state.cpp:39-46).
GPR_D void Sigma0(const double *Q, const Prim<false> &s, double *S) {
  sigma_col<false>(Q, s, 0, S);
  S[0] = s.p - S[0];
  S[1] = -S[1];
  S[2] = -S[2];
}

// d sigma(:, 0) / d rho and d sigma(:, 0) / dA (variables/state.cpp:43-56,
// energy/derivatives.cpp).
GPR_D void dsigma0(const double *Q, const Prim<false> &s, const DevPar &P, double *sr,
                   double *Pi1) {
  double r = s.r;
  sigma_col<false>(Q, s, 0, sr);
  double f = (1.0 + P.beta) * s.ir;  // 1 / rho + (d cs2 / d rho) / cs2
  for (int i = 0; i < 3; i++)
    sr[i] *= f;
  const double *A = Q + 5;
  const double G0[3] = {s.G[0], s.G[3], s.G[4]}, w = -r * s.cs2;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      double ret = (j == 0 ? 2.0 : 1.0) * s.AdG[3 * i + j];
      ret = fma(1.0 / 3.0 * A[3 * i], G0[j], ret);
      Pi1[3 * j + i] = w * fma(s.G[0], A[3 * i + j], ret);
    }
}

// c_0^2 (waves/speeds.cpp:8-18).
GPR_D double c0sq_of(const Prim<false> &s, const DevPar &P) {
  double r = s.r, G = s.e.G, dG = s.e.dG, rG = r * G, irG = s.irG;
  double dedrho = s.e.der - (s.e.dpr * rG + (G + r * dG) * (s.p - s.e.pr)) * (irG * irG);
  double iG = r * irG;
  double dcs2 = P.beta * s.ir * s.cs2;
  double dC0 = (1.0 - P.beta * iG) * dcs2 + P.beta * (iG * iG) * dG * s.cs2;
  double dEdr = dedrho + dC0 * 0.25 * s.devGsq;
  return (s.p * (s.ir * s.ir) - dEdr) * rG;
}

// The first three columns of riemann_constraints (riemann.cpp:79-154) for
// the non-thermal system; rows 0-4 are X, rows 11-13 -sgn Y0 Xi1 X, the rest
// zero (the other columns multiply zero coefficients in star_stepper).
// Rx is [5][3], Ry is [3][3].
//
// X solves the reference's 5 x 5 system: with y = its rows 2-4 (the
// distortion's first column), the two lower rows say (rho, p) = BA y, BA =
// (rho, 0, 0; sigma0 - rho sigma_r + rho c0^2 e0) A^-1, whatever regular
// matrix the reference multiplies them by, and the upper ones become (-Pi1 -
// sigma_r BA0 + e0 BA1) y = I: one 3 x 3 inverse, whose determinant is that of
// Pi1 times that of the reference's 2 x 2 factor Z.
GPR_D bool constraints(const double *Q, const Prim<false> &s, double sgn, const DevPar &P,
                       double *Rx, double *Ry) {
  const double r = s.r, ir = s.ir;
  const double *A = Q + 5;
  const double c02 = c0sq_of(s, P);
  // the reference takes the root (waves/speeds.cpp:17): a negative square, or a
  // NaN, makes its whole step NaN, although the shear part may keep the
  // spectrum of Xi real and positive
  if (!(c02 >= 0.0))
    return false;
  double sr[3], Pi1[9], sg[3];
  dsigma0(Q, s, P, sr, Pi1);
  sigma_col<false>(Q, s, 0, sg);
  const double x1[3] = {fma(r, c02, fma(-r, sr[0], sg[0])), fma(-r, sr[1], sg[1]),
                        fma(-r, sr[2], sg[2])};
  double At[9], BA[6];  // BA^T = A^-T (rho e0, x1)
  for (int i = 0; i < 3; i++) {
    for (int j = 0; j < 3; j++)
      At[3 * i + j] = A[3 * j + i];
    BA[2 * i] = i == 0 ? r : 0.0;
    BA[2 * i + 1] = x1[i];
  }
  if (!gauss<3, 2>(At, BA))
    return false;
  double N[9], y[9];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      N[3 * i + j] = fma(-sr[i], BA[2 * j], -Pi1[3 * i + j]);
      if (i == 0)
        N[j] += BA[2 * j + 1];
      y[3 * i + j] = i == j ? 1.0 : 0.0;
    }
  if (!gauss<3, 3>(N, y))
    return false;
  for (int j = 0; j < 3; j++) {
    for (int i = 0; i < 2; i++)
      Rx[3 * i + j] = BA[i] * y[j] + BA[2 + i] * y[3 + j] + BA[4 + i] * y[6 + j];
    for (int i = 0; i < 3; i++)
      Rx[3 * (2 + i) + j] = y[3 * i + j];
  }
  // Xi1 Xi2 and Xi1 X of system/eig.cpp:8-53 along x, without Xi1's and Xi2's
  // zeros: Xi1 = (-sigma_r, e0, -Pi1) / rho
  double Xi[9], Y0[9], X1X[9];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      double t = Pi1[3 * i] * A[j] + Pi1[3 * i + 1] * A[3 + j] + Pi1[3 * i + 2] * A[6 + j];
      double u = Pi1[3 * i] * y[j] + Pi1[3 * i + 1] * y[3 + j] + Pi1[3 * i + 2] * y[6 + j];
      u = fma(sr[i], Rx[j], u);
      if (i == 0) {
        t -= x1[j];
        u -= Rx[3 + j];
      }
      Xi[3 * i + j] = j == 0 ? fma(-ir, t, -sr[i]) : -ir * t;
      X1X[3 * i + j] = -ir * u;
    }
  if (!spectrum_positive(Xi) || !inv_sqrt3(Xi, Y0))
    return false;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      Ry[3 * i + j] = -sgn * (Y0[3 * i] * X1X[j] + Y0[3 * i + 1] * X1X[3 + j] +
                              Y0[3 * i + 2] * X1X[6 + j]);
  return true;
}

// Cvec_to_Pvec + P += R c + Pvec_to_Cvec (functions/vectors.cpp:85-154,
// riemann.cpp:191-200) for the non-thermal layout
// P = [rho, p, A(:,0), A(:,1), A(:,2), v, phi].
GPR_D void apply_correction(double *Q, const Prim<false> &s, const double *Rx,
                            const double *Ry, const double *cc, const DevPar &P) {
  double Pv[14];
  Pv[0] = Q[0];
  Pv[1] = s.p;
  for (int j = 0; j < 3; j++)
    for (int i = 0; i < 3; i++)
      Pv[2 + 3 * j + i] = Q[5 + 3 * i + j];
  for (int i = 0; i < 3; i++)
    Pv[11 + i] = Q[2 + i] * s.ir;
  for (int k = 0; k < 5; k++)
    Pv[k] += Rx[3 * k] * cc[0] + Rx[3 * k + 1] * cc[1] + Rx[3 * k + 2] * cc[2];
  for (int k = 0; k < 3; k++)
    Pv[11 + k] += Ry[3 * k] * cc[0] + Ry[3 * k + 1] * cc[1] + Ry[3 * k + 2] * cc[2];
  double r = Pv[0], p = Pv[1];
  Q[0] = r;
  double A[9];
  for (int j = 0; j < 3; j++)
    for (int i = 0; i < 3; i++)
      A[3 * i + j] = Pv[2 + 3 * j + i];
  for (int k = 0; k < 9; k++)
    Q[5 + k] = A[k];
  double v0 = Pv[11], v1 = Pv[12], v2 = Pv[13];
  Q[2] = r * v0;
  Q[3] = r * v1;
  Q[4] = r * v2;
  // total_energy (energy/eos.cpp:43-47)
  const double ir = rcp64(r);
  EosRho e = eos_rho(r, ir, P);
  double C0q = P.b02q;  // C_0 / 4, as prim() forms it
  if (P.has_beta) {
    const double cs2 = P.b02 * pow(r * P.ir0, P.beta);
    C0q = 0.25 * ((P.EOS == 1 ? (1.0 - P.beta / e.G) : P.C0f) * cs2);
  }
  double G00 = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
  double G11 = A[3] * A[3] + A[4] * A[4] + A[5] * A[5];
  double G22 = A[6] * A[6] + A[7] * A[7] + A[8] * A[8];
  double G01 = A[0] * A[3] + A[1] * A[4] + A[2] * A[5];
  double G02 = A[0] * A[6] + A[1] * A[7] + A[2] * A[8];
  double G12 = A[3] * A[6] + A[4] * A[7] + A[5] * A[8];
  double t = (G00 + G11 + G22) * (1.0 / 3.0);
  double dg = (G00 - t) * (G00 - t) + (G11 - t) * (G11 - t) + (G22 - t) * (G22 - t) +
              2.0 * (G01 * G01 + G02 * G02 + G12 * G12);
  const double irG = P.EOS == 1 ? P.iG : ir * P.iG;
  double E = e.er + (p - e.pr) * irG + 0.5 * (v0 * v0 + v1 * v1 + v2 * v2) + C0q * dg;
  Q[1] = r * E;
}

// left_star_state (riemann.cpp:203-233): the left star state of the
// interface Riemann problem between QL (material PL) and QR (material PR)
// along the unit normal n: at most ten linearised steps (star_stepper,
// riemann.cpp:156-201, slip_bcs, conditions.cpp:31-64), each after a half
// step dt/2 of the stiff relaxation, until check_star_convergence
// (riemann.cpp:26-77) holds; the input is returned if a NaN appears.  The
// level set entry (index 14) is carried through unchanged.
//
// Two neighbouring lanes work on one problem, the even one on the left
// state and the odd one on the right (each lane's Q0, P its own; EOS, rho0
// and b02 of the other side's material): the sides meet in one normal
// velocity and stress per step.  An interface of the 800 x 400 bubble has
// ~1000 problems, a few warps for 608 schedulers, so a launch lasts as long
// as one problem's chain of FP64 instructions (64 cycles each): 1.2 ms with
// one lane per problem, eliminations with a division per entry, two more of
// them and a matrix root of 18 inverses per side and step; 0.27 ms now.  Every lane of the
// warp calls it (live: the pair has a problem); the even lane writes out.
constexpr double STAR_TOL = 1e-8;  // options.h:22
GPR_D void left_star_pair(const double *Q0, const DevPar &P, int oEOS, double orho0, double ob02,
                          double dt, const double n[2], int nd, bool live, double *out) {
  const bool right = threadIdx.x & 1;
  const bool two = (right ? P.EOS : oEOS) > -1;  // the right side is a material
  const bool work = live && (two || !right);
  const double r0 = fmin(P.rho0, orho0), b02 = fmin(P.b02, ob02);
  double Q[15], R[3][3];
  for (int k = 0; k < 15; k++)
    Q[k] = work ? Q0[k] : 0.0;
  rotation(n, nd, R);
  rotate(Q, R);
  bool open = live, bad = false;
  for (int count = 0; count < 10; count++) {
    double S[3] = {0.0, 0.0, 0.0}, y = 0.0;
    if (open && work) {
      Prim<false> s;
      prim<false>(Q, P, s);
      Sigma0(Q, s, S);
      y = s.v[0];
    }
    const double So = __shfl_xor_sync(0xffffffffu, S[0], 1);
    const double yo = __shfl_xor_sync(0xffffffffu, y, 1);
    bool conv;
    if (two)
      conv = fabs(S[0] - So) < STAR_TOL * (b02 * r0) && fabs(y - yo) < STAR_TOL * sqrt64(b02);
    else
      conv = fmax(fabs(S[0]), fmax(fabs(S[1]), fabs(S[2]))) < STAR_TOL * (P.b02 * P.rho0);
    // (the left lane decides: with one material only it has the stress)
    conv = (__ballot_sync(0xffffffffu, conv) >> (threadIdx.x & 30u)) & 1u;
    open = open && !conv;
    if (!__any_sync(0xffffffffu, open))
      break;
    const bool step = open && work;
    double Rx[15], Ry[9], x[3] = {0.0, 0.0, 0.0}, d = 0.0, Ry0 = 0.0;
    bool ok = true;
    Prim<false> s;
    y = 0.0;
    if (step) {
      // ode_stepper_analytic (relaxation/analytic.cpp:152-161), no heat flux
      Q[2] += P.dp0 * dt * 0.5;
      Q[3] += P.dp1 * dt * 0.5;
      Q[4] += P.dp2 * dt * 0.5;
      ode_distortion(Q, dt * 0.5, P);
      prim<false>(Q, P, s);
      ok = constraints(Q, s, right ? -1.0 : 1.0, P, Rx, Ry);
      Sigma0(Q, s, x);
      y = s.v[0];
      // row 11 of the constraint matrices (the normal velocity)
      if (ok) {
        d = Ry[0] * x[0] + Ry[1] * x[1] + Ry[2] * x[2];
        Ry0 = Ry[0];
      }
    }
    const double yq = __shfl_xor_sync(0xffffffffu, y, 1);
    const double dq = __shfl_xor_sync(0xffffffffu, d, 1);
    const double Rq = __shfl_xor_sync(0xffffffffu, Ry0, 1);
    const bool okq = __shfl_xor_sync(0xffffffffu, (int)ok, 1);
    if (open && !(ok && okq)) {
      bad = true;
      open = false;
    }
    if (open && work) {
      double cc[3] = {-x[0], -x[1], -x[2]};
      if (two) {
        // (yR - yL + dL - dR) / (RL - RR), the same number from either side
        const double num = right ? (y - yq) + (dq - d) : (yq - y) + (d - dq);
        cc[0] = num / (right ? Rq - Ry0 : Ry0 - Rq) - x[0];
      }
      apply_correction(Q, s, Rx, Ry, cc, P);
    }
  }
  if (right || !live)
    return;
  for (int k = 0; k < 15; k++)
    bad = bad || isnan(Q[k]);
  if (bad) {
    for (int k = 0; k < 15; k++)
      out[k] = Q0[k];
    return;
  }
  double RT[3][3];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      RT[i][j] = R[j][i];
  rotate(Q, RT);
  for (int k = 0; k < 15; k++)
    out[k] = Q[k];
}

// ===========================================================================
// Boundary fill (multi/fill.cpp:96-235).

// One boundary cell (intMask == 1: the first ghost cell outside material
// mat) and where its fill reads and writes.
struct BPlan {
  int c;       // the cell
  int R;       // probe on the far side of the interface (QR)
  int ql;      // cell QL is read from
  int wi;      // interface cell also written (-1: none)
  int miR;     // material of QR
  int pad;
  double n[2]; // normal (axis-aligned by the fallback branch)
};

// get_material_index (functions/vectors.cpp:24-31) from the level set entry.
template <int V> GPR_D int mat_of(const double *grid, long c) {
  return grid[c * V + V - 1] >= 0.0 ? 1 : 0;
}

// Unit normal of dphi row c (normal, multi/functions.cpp:14); false when it
// is not finite.
GPR_D bool unit_normal(const double *dphi, long c, int nd, double n[2]) {
  if (nd == 1) {
    double g = dphi[c];
    double s = __dsqrt_rn(mul(g, g));
    n[0] = dvd(g, s);
    n[1] = 0.0;
    return isfinite(n[0]);
  }
  double g0 = dphi[2 * c], g1 = dphi[2 * c + 1];
  double s = __dsqrt_rn(add(mul(g0, g0), mul(g1, g1)));
  n[0] = dvd(g0, s);
  n[1] = dvd(g1, s);
  return isfinite(n[0]) && isfinite(n[1]);
}

// Plans every boundary cell: boundary_inds (fill.cpp:96-132) and the choice
// of QL in fill_boundary_inner (fill.cpp:134-198).  Cells whose fill would
// read outside the grid in the reference are counted in err[1] and left
// unfilled.  lastw[x] collects the largest boundary cell writing x.
template <int V>
__global__ void k_plan(const double *__restrict__ phi, const double *__restrict__ dphi,
                       const int32_t *__restrict__ im, const double *__restrict__ grid,
                       int mat, Grid g,
                       BPlan *__restrict__ plan, int *__restrict__ nplan,
                       int32_t *__restrict__ pidx, int32_t *__restrict__ lastw,
                       int *__restrict__ err, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell || im[c] != 1)
    return;
  int i = g.nd == 1 ? (int)c : (int)(c / g.ny), j = g.nd == 1 ? 0 : (int)(c % g.ny);
  double n[2];
  if (!unit_normal(dphi, c, g.nd, n)) {
    atomicAdd(&err[1], 1);
    return;
  }
  double phii = phi[c];
  int vi[2], vl[2], vr[2];
  int ind2[2] = {i, j};
  for (int k = 0; k < g.nd; k++) {
    double h = k == 0 ? g.dx : g.dy;
    double xp = mul(add((double)ind2[k], 0.5), h);
    double xi = sub(xp, mul(phii, n[k]));
    double hn = mul(mul(1.0, h), n[k]);
    vi[k] = (int)dvd(xi, h);
    vl[k] = (int)dvd(sub(xi, hn), h);
    vr[k] = (int)dvd(add(xi, hn), h);
  }
  long interf = g.nd == 1 ? vi[0] : (long)vi[0] * g.ny + vi[1];
  long L = g.nd == 1 ? vl[0] : (long)vl[0] * g.ny + vl[1];
  long R = g.nd == 1 ? vr[0] : (long)vr[0] * g.ny + vr[1];
  if (interf < 0 || interf >= g.ncell || L < 0 || L >= g.ncell || R < 0 || R >= g.ncell) {
    atomicAdd(&err[1], 1);
    return;
  }
  long ql;
  if (mat_of<V>(grid, interf) == mat) {
    ql = interf;
  } else if (mat_of<V>(grid, L) == mat) {
    ql = L;
  } else {
    if (g.nd == 1) {
      atomicAdd(&err[1], 1);
      return;
    }
    int Li[2] = {i, j};
    long Lind;
    int n0 = (n[0] > 0) - (n[0] < 0), n1 = (n[1] > 0) - (n[1] < 0);
    if (fabs(n[0]) > fabs(n[1])) {
      Li[0] -= n0;
      Lind = (long)Li[0] * g.ny + Li[1];
      if (Lind >= 0 && Lind < g.ncell && mat_of<V>(grid, Lind) == mat) {
        n[0] = n0;
        n[1] = 0.0;
      } else {
        Li[0] += n0;
        Li[1] -= n1;
        Lind = (long)Li[0] * g.ny + Li[1];
        n[0] = 0.0;
        n[1] = n1;
      }
    } else {
      Li[1] -= n1;
      Lind = (long)Li[0] * g.ny + Li[1];
      if (Lind >= 0 && Lind < g.ncell && mat_of<V>(grid, Lind) == mat) {
        n[0] = 0.0;
        n[1] = n1;
      } else {
        Li[0] -= n0;
        Li[1] += n1;
        Lind = (long)Li[0] * g.ny + Li[1];
        n[0] = n0;
        n[1] = 0.0;
      }
    }
    if (Lind < 0 || Lind >= g.ncell) {
      atomicAdd(&err[1], 1);
      return;
    }
    if (mat_of<V>(grid, Lind) == mat) {
      ql = Lind;
    } else {
      // neighbor_index(intMask, i, j, nx, ny, -1) (fill.cpp:76-94): the
      // last of left, right, down, up with intMask -1
      long indn = -1;
      if (i > 0 && im[c - g.ny] == -1)
        indn = c - g.ny;
      if (i < g.nx - 1 && im[c + g.ny] == -1)
        indn = c + g.ny;
      if (j > 0 && im[c - 1] == -1)
        indn = c - 1;
      if (j < g.ny - 1 && im[c + 1] == -1)
        indn = c + 1;
      if (indn < 0) {
        atomicAdd(&err[1], 1);
        return;
      }
      ql = indn;
    }
  }
  int k = atomicAdd(nplan, 1);
  BPlan b;
  b.c = (int)c;
  b.R = (int)R;
  b.ql = (int)ql;
  b.wi = mat_of<V>(grid, interf) != mat ? (int)interf : -1;
  b.miR = mat_of<V>(grid, R);
  b.pad = 0;
  b.n[0] = n[0];
  b.n[1] = n[1];
  plan[k] = b;
  pidx[c] = k;
  atomicMax(&lastw[c], (int)c);
  if (b.wi >= 0)
    atomicMax(&lastw[b.wi], (int)c);
}

// For each plan entry, the entry whose fill last wrote its QR cell earlier
// in the reference's (i, j) sweep (-1: QR is the original state), and its
// level in that dependency chain.
__global__ void k_plan_deps(const BPlan *__restrict__ plan, const int *__restrict__ nplan,
                            const int32_t *__restrict__ pidx,
                            const int32_t *__restrict__ lastw, int32_t *__restrict__ dep,
                            const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  int B = *nplan;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < B; k += gridDim.x * blockDim.x) {
    int c = plan[k].c, R = plan[k].R;
    int w = lastw[R];
    int dk = -1;
    if (w >= 0 && w < c) {
      dk = pidx[w];
    } else if (w >= c) {
      // a later (or this) cell writes R too: scan for the last earlier one
      int best = -1;
      for (int q = 0; q < B; q++) {
        int cq = plan[q].c;
        if (cq < c && cq > best && (cq == R || plan[q].wi == R))
          best = cq;
      }
      dk = best >= 0 ? pidx[best] : -1;
    }
    dep[k] = dk;
  }
}

__global__ void k_plan_levels(const int *__restrict__ nplan, const int32_t *__restrict__ dep,
                              int32_t *__restrict__ level, int *__restrict__ maxlevel,
                              const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  int B = *nplan;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < B; k += gridDim.x * blockDim.x) {
    int L = 0, q = dep[k];
    while (q >= 0 && L < B) {
      L++;
      q = dep[q];
    }
    level[k] = L;
    if (L > 0)
      atomicMax(maxlevel, L);
  }
}

// The star state of plan entry k, by two lanes (left_star_pair): every lane of
// the warp calls it, live where the pair has an entry.
template <int V>
GPR_D void solve_plan(int k, bool live, const BPlan *plan, const int32_t *dep,
                      const double *grid, double *star, const DevPar &P0, const DevPar &P1,
                      int mat, double dt, int nd) {
  static_assert(V == 15, "the ghost fill is for the viscous one-level-set layout");
  const BPlan &b = plan[live ? k : 0];
  const bool right = threadIdx.x & 1;
  const int miR = live ? b.miR : 0, dk = live ? dep[k] : -1;
  const DevPar &P = (right ? miR : mat) == 0 ? P0 : P1;
  const DevPar &O = (right ? mat : miR) == 0 ? P0 : P1;
  double Q[V], n[2] = {1.0, 0.0};
  if (live) {
    const double *src = grid + (long)(right ? b.R : b.ql) * V;
    for (int v = 0; v < V; v++)
      Q[v] = right && dk >= 0 && v < V - 1 ? star[(long)dk * V + v] : src[v];
    n[0] = b.n[0];
    n[1] = b.n[1];
  }
  left_star_pair(Q, P, O.EOS, O.rho0, O.b02, dt, n, nd, live, star + (long)(live ? k : 0) * V);
}

// Star states of the plan entries on level 0 (all independent).
template <int V>
__global__ void __launch_bounds__(32)
    k_star_level0(const BPlan *__restrict__ plan, const int *__restrict__ nplan,
                  const int32_t *__restrict__ dep, const int32_t *__restrict__ level,
                  const double *grid, double *star, DevPar P0, DevPar P1, int mat, double dt,
                  const double *__restrict__ dt_dev, int nd, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  if (dt_dev)
    dt = *dt_dev;
  const int B = *nplan;
  for (int k0 = blockIdx.x * 16; k0 < B; k0 += gridDim.x * 16) {
    const int k = k0 + (int)(threadIdx.x >> 1);
    const bool live = k < B && level[k] == 0;
    if (__any_sync(0xffffffffu, live))
      solve_plan<V>(k, live, plan, dep, grid, star, P0, P1, mat, dt, nd);
  }
}

// Deeper levels, in order, in one block (rare: only where a boundary cell's
// far-side probe was filled earlier in the sweep).
template <int V>
__global__ void __launch_bounds__(64)
    k_star_levels(const BPlan *__restrict__ plan, const int *__restrict__ nplan,
                  const int32_t *__restrict__ dep, const int32_t *__restrict__ level,
                  const int *__restrict__ maxlevel, const double *grid, double *star, DevPar P0,
                  DevPar P1, int mat, double dt, const double *__restrict__ dt_dev, int nd,
                  const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  if (dt_dev)
    dt = *dt_dev;
  const int B = *nplan, ML = *maxlevel;
  for (int L = 1; L <= ML; L++) {
    for (int k0 = 0; k0 < B; k0 += 32) {
      const int k = k0 + (int)(threadIdx.x >> 1);
      const bool live = k < B && level[k] == L;
      if (__any_sync(0xffffffffu, live))
        solve_plan<V>(k, live, plan, dep, grid, star, P0, P1, mat, dt, nd);
    }
    __syncthreads();
  }
}

// Every written cell takes the star state of its last writer in the sweep;
// the level set entry keeps the grid's value (fill.cpp:194-197).
template <int V>
__global__ void k_scatter(const BPlan *__restrict__ plan, const int *__restrict__ nplan,
                          const int32_t *__restrict__ lastw, const double *__restrict__ star,
                          double *__restrict__ grid, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  int B = *nplan;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < B; k += gridDim.x * blockDim.x) {
    int c = plan[k].c, wi = plan[k].wi;
    if (lastw[c] == c)
      for (int v = 0; v < V - 1; v++)
        grid[(long)c * V + v] = star[(long)k * V + v];
    if (wi >= 0 && lastw[wi] == c)
      for (int v = 0; v < V - 1; v++)
        grid[(long)wi * V + v] = star[(long)k * V + v];
  }
}

// ===========================================================================
// Layered fill (fill_neighbor_cells, multi/fill.cpp:237-328): layer N0 + 1
// is every cell with intMask 0 (or -2 in 2D) next to a layer-N0 cell.

struct Layer {
  const int32_t *m;  // intMask before this layer
  Grid g;
  int N0;
  GPR_D bool open(long x) const {
    int v = m[x];
    return v == 0 || (g.nd == 2 && v == -2);
  }
  // is x in this layer; indn = the reference's neighbour index (the last
  // match in the order left, right, down, up)
  GPR_D bool in(long x, long &indn) const {
    indn = -1;
    if (!open(x))
      return false;
    if (g.nd == 1) {
      int i = (int)x;
      if (i > 0 && m[x - 1] == N0)
        indn = x - 1;
      if (i < g.nx - 1 && m[x + 1] == N0)
        indn = x + 1;
      return indn >= 0;
    }
    int i = (int)(x / g.ny), j = (int)(x % g.ny);
    if (i > 0 && m[x - g.ny] == N0)
      indn = x - g.ny;
    if (i < g.nx - 1 && m[x + g.ny] == N0)
      indn = x + g.ny;
    if (j > 0 && m[x - 1] == N0)
      indn = x - 1;
    if (j < g.ny - 1 && m[x + 1] == N0)
      indn = x + 1;
    return indn >= 0;
  }
};

// One layer.  In the reference's sweep a new cell copies the cell one step
// towards the interface along its normal if that cell's mask is >= 1 at
// that moment, else the layer-N0 neighbour it was reached from; cells of
// this layer visited earlier in the sweep already hold their copies, so a
// copy from one of them is followed to where it copied from.
template <int V>
__global__ void k_layer(double *__restrict__ grid, const int32_t *__restrict__ mprev,
                        int32_t *__restrict__ mnext, const double *__restrict__ dphi, Grid g,
                        int N0, int *__restrict__ err, const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= g.ncell)
    return;
  Layer Ly{mprev, g, N0};
  long indn;
  if (!Ly.in(c, indn)) {
    mnext[c] = mprev[c];
    return;
  }
  mnext[c] = mprev[c] == -2 ? -2 : N0 + 1;  // isolated cells return to -2
  long x = c, xn = indn, src = -1;
  for (int hops = 0; hops < 4096; hops++) {
    double n[2];
    long nind = -1;
    if (unit_normal(dphi, x, g.nd, n)) {
      int i = g.nd == 1 ? (int)x : (int)(x / g.ny), j = g.nd == 1 ? 0 : (int)(x % g.ny);
      int ind2[2] = {i, j}, ni[2] = {0, 0};
      for (int k = 0; k < g.nd; k++) {
        double h = k == 0 ? g.dx : g.dy;
        double xc = mul(add((double)ind2[k], 0.5), h);
        ni[k] = (int)dvd(sub(xc, mul(h, n[k])), h);
      }
      nind = g.nd == 1 ? ni[0] : (long)ni[0] * g.ny + ni[1];
    }
    bool off = nind < 0 || nind >= g.ncell;
    if (off) {
      atomicAdd(&err[2], 1);
      src = xn;
      break;
    }
    if (nind == x) {  // copies itself: keeps its own value
      src = x;
      break;
    }
    long nn;
    if (nind < x && Ly.in(nind, nn)) {  // filled earlier in this layer
      x = nind;
      xn = nn;
      continue;
    }
    src = mprev[nind] >= 1 ? nind : xn;
    break;
  }
  if (src < 0) {
    atomicAdd(&err[2], 1);
    return;
  }
  if (src != c)
    for (int v = 0; v < V - 1; v++)
      grid[c * V + v] = grid[src * V + v];
}

// Update mask of material mat (fill.cpp:364-365).
__global__ void k_mat_mask(const double *__restrict__ phi, const int32_t *__restrict__ im,
                           uint8_t *__restrict__ mask, long ncell,
                           const double *__restrict__ clk) {
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  int m = im[c];
  mask[c] = (phi[c] <= 0.0 && m != -2) || m == 1;
}

// ===========================================================================
// Merge, CFL and renormalisation over material grids.

// make_u (solvers/iterator.cpp:12-42): the level set averaged over the
// grids that updated the cell, the rest of the state from the grid of the
// cell's material (zero for a vacuum).
template <int V>
__global__ void k_make_u(double *__restrict__ u, const double *__restrict__ grids,
                         const uint8_t *__restrict__ masks, long ncell, int nmat, int eos0,
                         int eos1, const double *__restrict__ dt_dev) {
  if (dt_dev && *dt_dev == 0.0)
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  double s = 0.0, cnt = 0.0;
  for (int m = 0; m < nmat; m++)
    if (masks[(long)m * ncell + c]) {
      s += grids[((long)m * ncell + c) * V + V - 1];
      cnt += 1.0;
    }
  if (cnt > 0.0)
    u[c * V + V - 1] = s / cnt;
  int mi = u[c * V + V - 1] >= 0.0 ? 1 : 0;
  int eos = mi == 0 ? eos0 : eos1;
  for (int v = 0; v < V - 1; v++)
    u[c * V + v] = eos > -1 ? grids[((long)mi * ncell + c) * V + v] : 0.0;
}

// timestep (solvers/iterator.cpp:54-83): max over the masked cells of one
// material grid, accumulated over materials in *out.
template <class L>
__global__ void __launch_bounds__(256)
    k_cfl_max_masked(const double *__restrict__ u, const uint8_t *__restrict__ mask, long ncell,
                     int nd, double dx, double dy, unsigned long long *__restrict__ out,
                     DevPar P, const double *__restrict__ clk) {
  constexpr int V = L::V;
  if (clk && clk[0] >= clk[2])
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double m = 0.0;
  if (c < ncell && mask[c]) {
    double q[V];
    for (int k = 0; k < V; k++)
      q[k] = u[c * V + k];
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(q, P, s);
    double tmp = max_abs_eigs<L::THERMAL>(q, s, 0, P) / dx;
    if (nd == 2)
      tmp += max_abs_eigs<L::THERMAL>(q, s, 1, P) / dy;
    if (tmp > m)
      m = tmp;
  }
  for (int o = 16; o > 0; o >>= 1)
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double sm[8];
  if ((threadIdx.x & 31) == 0)
    sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++)
      b = fmax(b, sm[w]);
    atomicMax(out, (unsigned long long)__double_as_longlong(b));
  }
}

// renorm_distortion (solvers/utils.cpp:6-23) with each cell's material
// from its level set.
template <int V>
__global__ void k_renorm_multi(double *__restrict__ u, long ncell, double r00, double r01,
                               int eos0, int eos1, const double *__restrict__ dt_dev) {
  if (dt_dev && *dt_dev == 0.0)
    return;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  double *q = u + c * V;
  int mi = q[V - 1] >= 0.0 ? 1 : 0;
  if ((mi == 0 ? eos0 : eos1) <= -1)
    return;
  double r = q[0];
  if (r > 0) {
    double A[9];
    for (int k = 0; k < 9; k++)
      A[k] = q[5 + k];
    double f = cbrt(r / ((mi == 0 ? r00 : r01) * det3(A)));
    for (int k = 0; k < 9; k++)
      q[5 + k] = A[k] * f;
  }
}

// Pointwise left_star_state for tests and the system.multi binding.
template <int V>
__global__ void k_star_pointwise(const double *QL, const double *QR,
                                 const double *__restrict__ nrm, double *out,
                                 long count, int nd, double dt, DevPar PL, DevPar PR) {
  const long k = blockIdx.x * (long)(blockDim.x / 2) + (threadIdx.x >> 1);
  const bool live = k < count, right = threadIdx.x & 1;
  const long kk = live ? k : 0;
  double n[2] = {nrm[kk * nd], nd == 2 ? nrm[kk * nd + 1] : 0.0};
  const DevPar &P = right ? PR : PL, &O = right ? PL : PR;
  left_star_pair((right ? QR : QL) + kk * V, P, O.EOS, O.rho0, O.b02, dt, n, nd, live,
                 out + kk * V);
}

}  // namespace multi
}  // namespace gpr
