// gpr_kernels.cuh - the ADER-WENO step kernels (N = 2), templated on the
// variable layout (THERMAL, LSET).  Host-side launchers live in gpr_capi.cu.
#pragma once

#include "gpr_consts.cuh"
#include "gpr_device.cuh"

namespace gpr {

constexpr double LAMS = 1.0;       // WENO side-stencil weight (options.h:24)
constexpr double WENO_EPS = 1e-14; // options.h:26

template <bool TH, int LS> struct Layout {
  static constexpr bool THERMAL = TH;
  static constexpr int LSET = LS;
  static constexpr int V = 14 + (TH ? 3 : 0) + LS;
};

// ---------------------------------------------------------------------------
// Batched form: many independent 1D grids (instances) of uneven sizes, each
// with its own material and its own clock, packed one after another.  For
// instance k with nx_k interior cells the packed index spaces are
//   u  cells   off_u[k]  .. off_u[k]  + nx_k      (off_u[k+1] = off_u[k] + nx_k)
//   ub cells   off_ub[k] .. off_ub[k] + nx_k + 2N (= off_u[k] + 2N k)
//   predictor  off_b[k]  .. off_b[k]  + nx_k + 2  (= off_u[k] + 2 k)
//   faces      off_f[k]  .. off_f[k]  + nx_k + 1  (= off_u[k] + k)
// and inst_* map every packed index to its instance.  clk[k] holds
// {t, dt, tf, cfl, count}; a finished instance has dt = 0 and its steps
// change nothing.
struct Batch {
  const DevPar *P;
  const int32_t *inst_u, *inst_ub, *inst_b, *inst_f;
  const int32_t *nx, *off_u, *off_ub, *off_b, *off_f, *bc;
  const double *idx;  // 1 / dx per instance
  double *clk;        // [ninst][5]
  int ninst;
};

// ---------------------------------------------------------------------------
// Boundary ghost cells (etc/grid.cpp:12-170).  One thread per (ghost row, k)
// of one axis; 2D runs the x pass over interior rows, then the y pass over
// all rows (corners are filled from x ghosts as in the reference).

GPR_D int bc_src_index(int code, int side, int i, int n) {
  // index into the interior line of length n for ghost i (0..N-1) of side
  if (code == GPR_BC_TRANSMISSIVE)
    return side == 0 ? 0 : n - 1;
  if (code == GPR_BC_PERIODIC)
    return side == 0 ? n - NN + i : i;
  return side == 0 ? NN - 1 - i : n - 1 - i;  // reflecting types
}

template <int V>
GPR_D double bc_value(int code, int d, int k, const double *src) {
  double x = src[k];
  switch (code) {
  case GPR_BC_SLIP:
  case GPR_BC_SYMMETRIC:
    if (k == 2 + d)
      x = -x;
    if (code == GPR_BC_SYMMETRIC && k >= 5 && k < 14) {
      int r = (k - 5) / 3, c = (k - 5) % 3;
      if (r == d)
        x = -x;
      if (c == d)
        x = -x;
    }
    break;
  case GPR_BC_STICK:
    if (k >= 2 && k < 5)
      x = -x;
    break;
  case GPR_BC_MOVING:
    if (k >= 2 && k < 5)
      x = -x;
    if (k == 2)
      x += 2.0 * src[0];
    if (k == 1) {
      double m = -src[2] + 2.0 * src[0];
      x += (m * m - src[2] * src[2]) / (2.0 * src[0]);
    }
    break;
  default:
    break;
  }
  return x;
}

// Copies interior u into ub (cell-major), one thread per (cell, var).
template <int V>
__global__ void k_fill_interior(const double *__restrict__ u, double *__restrict__ ub,
                                int nx, int ny, int nd) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  long total = (long)nx * ny * V;
  if (idx >= total)
    return;
  int k = idx % V;
  long c = idx / V;
  if (nd == 1) {
    ub[(c + NN) * V + k] = u[idx];
  } else {
    int i = c / ny, j = c % ny;
    ub[((long)(i + NN) * (ny + 2 * NN) + (j + NN)) * V + k] = u[idx];
  }
}

// 1D boundaries in one launch: ub[p] for p in 0..nx+2N-1, interior cells
// copied from u, ghost cells by the boundary rule from their source cell of u
// (the values k_fill_interior + k_ghosts give), one thread per (cell, var).
template <int V>
GPR_D double ub_value1d(const double *__restrict__ u, int p, int k, int nx, int bcl, int bcr) {
  if (p >= NN && p < nx + NN)
    return u[(long)(p - NN) * V + k];
  const int side = p >= nx + NN;
  const int i = side ? p - nx - NN : p;
  int code = side ? bcr : bcl;
  const int si = bc_src_index(code, side, i, nx);
  if (code == GPR_BC_PERIODIC)
    code = GPR_BC_TRANSMISSIVE;  // plain copy
  return bc_value<V>(code, 0, k, u + (long)si * V);
}
template <int V>
__global__ void k_boundaries1d(const double *__restrict__ u, double *__restrict__ ub, int nx,
                               int bcl, int bcr) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)(nx + 2 * NN) * V)
    return;
  ub[idx] = ub_value1d<V>(u, (int)(idx / V), (int)(idx % V), nx, bcl, bcr);
}

// Ghost rows along one axis.  For axis 0: lines are columns j (interior rows
// j+N of ub when nd == 2), for axis 1: lines are all ub rows i.
template <int V>
__global__ void k_ghosts(double *__restrict__ ub, int nx, int ny, int nd, int axis,
                         int bcl, int bcr) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int nline = nd == 1 ? 1 : (axis == 0 ? ny : nx + 2 * NN);
  long total = (long)nline * 2 * NN * V;
  if (idx >= total)
    return;
  int k = idx % V;
  long rest = idx / V;
  int g = rest % (2 * NN);  // ghost slot: 0..N-1 left, N..2N-1 right
  int line = rest / (2 * NN);
  int side = g >= NN;
  int i = side ? g - NN : g;
  int n = axis == 0 ? nx : ny;
  int code = side ? bcr : bcl;
  int si = bc_src_index(code, side, i, n);
  int gi = side ? i + n + NN : i;  // ghost position along the line
  long nyb = ny + 2 * NN;
  const double *src;
  double *dst;
  if (nd == 1) {
    src = ub + (long)(si + NN) * V;
    dst = ub + (long)gi * V;
  } else if (axis == 0) {
    long j = line + NN;
    src = ub + ((long)(si + NN) * nyb + j) * V;
    dst = ub + ((long)gi * nyb + j) * V;
  } else {
    long ii = line;
    src = ub + (ii * nyb + (si + NN)) * V;
    dst = ub + (ii * nyb + gi) * V;
  }
  if (code == GPR_BC_PERIODIC)
    code = GPR_BC_TRANSMISSIVE;  // plain copy
  dst[k] = bc_value<V>(code, axis, k, src);
}

// ---------------------------------------------------------------------------
// WENO (solvers/weno/weno.cpp:4-124).  One thread per (cell, variable):
// data rows d0[0], d0[sd], d0[2 sd] (cells i-1, i, i+1); writes the N = 2
// node values out[0], out[so].
//
// With two nodes a side stencil's polynomial is the line through two cell
// averages, w_n = b + (x_n - 1/2) dL with dL = b - a (dR = c - b on the
// right), and its oscillation indicator w^T SIG w the square of its slope,
// dL^2.  The blend of the two lines is the line of the blended slope, so a
// point takes 21 FP64 instructions where the products with the reference's
// matrices (weno_matrices.cpp:9-42) take 40; the slope is one rounded
// subtraction, which loses less on nearly constant data than those products.
// 512 x 512: k_weno2d 1.10 to 0.51 ms.
constexpr double WENO_X = 0.28867513459481288225;  // x_1 - 1/2 = 1 / (2 sqrt 3)
GPR_D void weno_line(double a, double b, double c, double *__restrict__ out, long so, int ind,
                     int nx, int gap) {
  const double dL = b - a, dR = c - b;
  double tL = fma(dL, dL, WENO_EPS), tR = fma(dR, dR, WENO_EPS);
  tL *= tL;
  tL *= tL;
  tL *= tL;
  tR *= tR;
  tR *= tR;
  tR *= tR;
  const bool useL = ind >= gap, useR = ind <= nx - gap - 1;
  // weights LAMS / tL, LAMS / tR normalised, i.e. tR / (tL + tR) and tL / (tL +
  // tR): one reciprocal where the reference takes three divisions
  static_assert(LAMS == 1.0, "equal side weights");
  double s = fma(dL, tR, dR * tL) * rcp64(tL + tR);
  // one-sided next to the edges; with neither side 0 / 0, as the reference
  if (!(useL && useR))
    s = useL ? dL : (useR ? dR : __longlong_as_double(0x7ff8000000000000LL));
  out[0] = fma(-WENO_X, s, b);
  out[so] = fma(WENO_X, s, b);
}
GPR_D void weno_point(const double *__restrict__ d0, long sd, double *__restrict__ out,
                      long so, int ind, int nx, int gap) {
  weno_line(d0[0], d0[sd], d0[2 * sd], out, so, ind, nx, gap);
}

// 1D: wh[i][a][k] for i in 0..nx+1 from ub rows i..i+2 (weno.cpp:75-81, 146)
template <int V>
__global__ void k_weno1d(double *__restrict__ wh, const double *__restrict__ ub, int ncb) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)ncb * V)
    return;
  int k = idx % V;
  int i = idx / V;
  weno_point(ub + (long)i * V + k, V, wh + (long)i * NN * V + k, V, i, ncb, 0);
}

// The same straight from u, for steps that need the extended grid for nothing
// else (one launch of ~3 us less).
template <int V>
__global__ void k_weno1d_u(double *__restrict__ wh, const double *__restrict__ u, int nx, int bcl,
                           int bcr) {
  const long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= (long)(nx + 2) * V)
    return;
  const int k = idx % V, i = idx / V;
  weno_line(ub_value1d<V>(u, i, k, nx, bcl, bcr), ub_value1d<V>(u, i + 1, k, nx, bcl, bcr),
            ub_value1d<V>(u, i + 2, k, nx, bcl, bcr), wh + (long)i * NN * V + k, V, i, nx + 2, 0);
}

// 2D, both sweeps in one launch, staged in shared memory: a block takes
// predictor row i (one of nx+2) and output columns j0 .. j0+jn-1 (jn <= tj).
// It loads the jn+2 ub columns of ub rows i, i+1, i+2 that the x sweep
// reads (each row segment is contiguous in the cell-major layout: 16-byte
// loads, with single doubles only at an unaligned start or end), runs the x
// sweep on them into a shared ux tile (node a = 0, 1 of each column), and
// the y sweep of its jn columns from that tile into wh.  Each point is
// weno_point with the reference's one-sided edges (weno.cpp:93-121); the
// x sweep's 2 edge columns of a tile are evaluated again by its neighbour
// tile.  ux never reaches global memory.  With a mask (a byte per predictor
// cell) only its cells are reconstructed, the others of wh are left as they
// are: for the two materials of an 800 x 400 bubble half of the work.
constexpr int WENO2_COLS = 64, WENO2_THREADS = 256;
template <int V>
__global__ void __launch_bounds__(WENO2_THREADS) k_weno2d(double *__restrict__ wh,
                                                         const double *__restrict__ ub,
                                                         int nxp, int nyp, int tj,
                                                         const uint8_t *__restrict__ mask) {
  constexpr int RS = WENO2_COLS * V;  // shared row stride (doubles)
  __shared__ double sub[3 * RS];
  __shared__ double sux[WENO2_COLS * NN * V];
  __shared__ uint8_t on[WENO2_COLS + 2];  // on[c + 2]: output column c is wanted
  const int nyb = nyp + 2 * (NN - 1);
  const int nbj = (nyp + tj - 1) / tj;
  const int i = blockIdx.x / nbj, j0 = (blockIdx.x % nbj) * tj;
  const int jn = min(tj, nyp - j0), nc = jn + 2;
  const int len = nc * V;
  const int tc = (int)threadIdx.x - 2;
  const bool want =
      tc >= 0 && tc < jn && (mask == nullptr || mask[(long)i * nyp + j0 + tc]);
  if (threadIdx.x < WENO2_COLS + 2)
    on[threadIdx.x] = want;
  if (!__syncthreads_or(want))
    return;
  // 1. stage ub rows i .. i+2, columns j0 .. j0+nc-1
  for (int r = 0; r < 3; r++) {
    const double *src = ub + ((long)(i + r) * nyb + j0) * V;
    const int off = (int)(((unsigned long long)src >> 3) & 1);  // src not 16-byte aligned
    const int npair = (off + len + 1) / 2;
    double *dst = sub + r * RS;
    for (int p = threadIdx.x; p < npair; p += WENO2_THREADS) {
      const int lo = 2 * p - off;  // element index of the pair's first double
      if (lo >= 0 && lo + 1 < len) {
        const double2 x = *reinterpret_cast<const double2 *>(src + lo);
        dst[lo] = x.x;
        dst[lo + 1] = x.y;
      } else {
        if (lo >= 0)
          dst[lo] = src[lo];
        if (lo + 1 >= 0 && lo + 1 < len)
          dst[lo + 1] = src[lo + 1];
      }
    }
  }
  __syncthreads();
  // 2. x sweep (weno.cpp:93-104) of the nc staged columns
  for (int e = threadIdx.x; e < len; e += WENO2_THREADS) {
    const int c = e / V, k = e % V;
    const int j = j0 + c;
    const int gap = (j < NN || j >= nyb - NN) ? NN : 0;
    if (on[c] | on[c + 1] | on[c + 2])  // read by output columns c - 2 .. c
      weno_point(sub + c * V + k, RS, sux + c * NN * V + k, V, i, nxp, gap);
  }
  __syncthreads();
  // 3. y sweep (weno.cpp:106-121) of the jn output columns
  const int gap = (i == 0 || i == nxp - 1) ? 1 : 0;
  for (int e = threadIdx.x; e < jn * NN * V; e += WENO2_THREADS) {
    const int k = e % V, a = (e / V) % NN, c = e / (NN * V);
    const int j = j0 + c;
    if (on[c + 2])
      weno_point(sux + (c * NN + a) * V + k, (long)NN * V,
                 wh + (((long)i * nyp + j) * NN * NN + a * NN) * V + k, V, j, nyp, gap);
  }
}

// Output columns per k_weno2d block: at most WENO2_COLS - 2, spread evenly
// over the row's blocks.
inline int weno2d_tile(int nyp) {
  const int nbj = (nyp + WENO2_COLS - 3) / (WENO2_COLS - 2);
  return (nyp + nbj - 1) / nbj;
}

// Sum an n-vector v over the G lanes of each aligned lane group (xor
// butterfly) and scatter the sum: afterwards lane r = lane % G holds
// elements r n/G .. (r + 1) n/G - 1 of the sum in v[0 .. n/G - 1].  At each
// level a lane keeps one half, chosen by its lane bit (a select: integer
// work), and adds the partner's copy of it, so a lane issues n/2 + n/4 + ...
// + n/G FP64 adds where a full butterfly issues n log2 G; on this GPU the
// FP64 cost is per warp instruction, whatever the active lanes.
template <int n, int G> struct GroupReduceScatter {
  static_assert(n % G == 0, "n a multiple of G");
  static GPR_D void run(double *v, int r) {
    if constexpr (G > 1) {
      constexpr int h = n / 2;
      const bool up = r & (G / 2);
#pragma unroll
      for (int j = 0; j < h; j++) {
        const double keep = up ? v[h + j] : v[j];
        const double send = up ? v[j] : v[h + j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, G / 2);
      }
      GroupReduceScatter<h, G / 2>::run(v, r);
    }
  }
};

// The face contributions kk (b + f) (left cell) and kk (b - f) (right cell)
// summed over the G quadrature lanes of a face (r = lane within the face)
// and written to out[0..V-1] / out[V..2V-1] by the lanes that hold them.  The
// two-point rule's weights are equal, so kk is the same on every lane of a face
// and multiplies the 2 V / G sums a lane ends with, not its 2 V terms.
template <int V, int G>
GPR_D void face_reduce_store(const double *b, const double *f, double kk, bool active,
                             bool valid, int r, double *out) {
  constexpr int NPR = (V + G - 1) / G;  // (b, f) pairs per lane after the scatter
  double v[2 * NPR * G];
#pragma unroll
  for (int k = 0; k < NPR * G; k++) {
    v[2 * k] = (active && k < V) ? b[k] : 0.0;
    v[2 * k + 1] = (active && k < V) ? f[k] : 0.0;
  }
  GroupReduceScatter<2 * NPR * G, G>::run(v, r);
  if (!valid)
    return;
#pragma unroll
  for (int p = 0; p < NPR; p++) {
    const int k = r * NPR + p;
    if (k < V) {
      out[k] = kk * (v[2 * p] + v[2 * p + 1]);
      out[V + k] = kk * (v[2 * p] - v[2 * p + 1]);
    }
  }
}

// The same sums applied to the state in place (interfs1 / interfs2 update u
// inside the face loop, fv.cpp:143-146, 217-222, 257-262): uL -= out[0..V-1]
// on the cell to the left of the face, uR -= out[V..2V-1] on the cell to its
// right (either may be null: no interior cell there).  Only for faces with
// face_on (the face's own activity: geometry and mask, not the lane's).
template <int V, int G>
GPR_D void face_reduce_apply(const double *b, const double *f, double kk, bool active,
                             bool face_on, int r, double *uL, double *uR) {
  constexpr int NPR = (V + G - 1) / G;
  double v[2 * NPR * G];
#pragma unroll
  for (int k = 0; k < NPR * G; k++) {
    v[2 * k] = (active && k < V) ? b[k] : 0.0;
    v[2 * k + 1] = (active && k < V) ? f[k] : 0.0;
  }
  GroupReduceScatter<2 * NPR * G, G>::run(v, r);
  if (!face_on)
    return;
#pragma unroll
  for (int p = 0; p < NPR; p++) {
    const int k = r * NPR + p;
    if (k < V) {
      if (uL)
        uL[k] = fma(-kk, v[2 * p] + v[2 * p + 1], uL[k]);
      if (uR)
        uR[k] = fma(-kk, v[2 * p] - v[2 * p + 1], uR[k]);
    }
  }
}

// Faces of one 2D face pass.  parity < 0: every face (i, j) of the
// (nx+1) x (ny+1) face grid of direction dir.  parity 0 / 1: only the faces
// whose index along dir has that parity; two such faces never share a cell,
// so a pass can update u in place without races, and the four passes
// (direction x parity) cover every face once.
struct Face2 {
  long fi;    // flat face index (i (ny + 1) + j)
  int i, j;   // predictor-cell indices of the face's left / lower cell
  bool valid;
};
GPR_HD long face2_count(int nx, int ny, int dir, int parity) {
  if (parity < 0)
    return (long)(nx + 1) * (ny + 1);
  return dir == 0 ? (long)((nx + 2 - parity) / 2) * (ny + 1)
                  : (long)(nx + 1) * ((ny + 2 - parity) / 2);
}
GPR_D Face2 face2_of(long face, int nx, int ny, int dir, int parity) {
  Face2 F;
  F.valid = face < face2_count(nx, ny, dir, parity);
  long e = F.valid ? face : 0;
  if (parity < 0) {
    F.i = e / (ny + 1);
    F.j = e % (ny + 1);
  } else if (dir == 0) {
    F.i = 2 * (int)(e / (ny + 1)) + parity;
    F.j = e % (ny + 1);
  } else {
    const int nfj = (ny + 2 - parity) / 2;
    F.i = e / nfj;
    F.j = 2 * (int)(e % nfj) + parity;
  }
  F.fi = (long)F.i * (ny + 1) + F.j;
  return F;
}
// The interior cells on either side of face (i, j) of direction dir, as
// pointers into u[nx][ny][V] (null where the side is a ghost cell).
GPR_D void face2_cells(double *u, int i, int j, int nx, int ny, int dir, int V, double *&uL,
                       double *&uR) {
  if (dir == 0) {
    uL = i >= 1 ? u + ((long)(i - 1) * ny + (j - 1)) * V : nullptr;
    uR = i <= nx - 1 ? u + ((long)i * ny + (j - 1)) * V : nullptr;
  } else {
    uL = j >= 1 ? u + ((long)(i - 1) * ny + (j - 1)) * V : nullptr;
    uR = j <= ny - 1 ? u + ((long)(i - 1) * ny + j) * V : nullptr;
  }
}

// ---------------------------------------------------------------------------
// Space-time DG predictor (solvers/dg/dg1.cpp:8-114, dg2.cpp:8-171).
//
// One thread per space-time node: NP = N^(d+1) consecutive lanes hold one
// cell (lane g = t N^d + s).  Spatial derivatives, the DG_DER flux term and
// the DG_U^-1 time coupling need the partner nodes' values, exchanged with
// warp shuffles (partners differ in one index: lane ^ bit).  Each iteration
// is the reference's Picard update q <- DG_U^-1 (Ww + dt R(q)) with its
// per-cell stopping rule |q1 - q0| <= dg_tol (1 + |q0|) (dg1.cpp:91-110).

// |x| as the bit pattern of a non-negative double; patterns above
// FP_INF_BITS are NaNs.
constexpr unsigned long long FP_INF_BITS = 0x7ff0000000000000ULL;
// growth of a cell's largest Picard update over its smallest that hands the
// cell to the Newton pass (k_predictor_picard): in general, and in a Newtonian
// fluid up to the caps below
constexpr float PICARD_DIVERGE = 1e3f, PICARD_GROWN = 31.6f;
// first iteration of the windows over which the rate of a cell's updates is
// taken, and the largest update over its threshold, extrapolated to the
// iteration cap in two windows running, that hands the cell over (log2)
constexpr int PICARD_WINDOW0 = 4;
constexpr float PICARD_HOPELESS = 16.6096f;  // 1e5
constexpr int PICARD_RATE_CAP = 50;  // the caps up to which both were measured
GPR_D unsigned long long fp_abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffULL;
}
// |x| in FP32 from its high word, truncated (relative error below 2^-20); 0
// below the FP32 range, F32_TOP from 2^127 on (infinities and NaNs included).
constexpr float F32_TOP = 1.7014118346046923e38f;  // 2^127
GPR_D float f32_abs_hi(double x) {
  int e = (__double2hiint(x) & 0x7fffffff) - (896 << 20);
  e = e < 0x00100000 ? 0 : (e > 0x0fe00000 ? 0x0fe00000 : e);
  return __int_as_float(e << 3);
}

template <int V>
GPR_D void shfl_vec(const double *src, double *dst, int lanemask) {
#pragma unroll
  for (int k = 0; k < V; k++)
    dst[k] = __shfl_xor_sync(0xffffffffu, src[k], lanemask);
}

// The system's pointwise residual at this thread's node, scaled:
//   r = sg (S(q) - B_x dq/dx [- B_y dq/dy] - dF/dx [- dG/dy]),
// the derivatives along the cell's node lines (S left out without SOURCE).
// The rhs of the Picard map is W_t W_s times this with sg = dt: W_t W_s (S - B
// dq) - W_t [W_j] DG_DER F / dx ..., since DG_DER(i, m) = W_i psi_m'(x_i).  With
// two nodes a line's derivative is the same difference quotient at both,
// (q1 - q0) / (x1 - x0), so it is one subtraction with the partner's value
// and the quotient goes into the coefficient (sign by the lane's end).
// hx, hy: 1 / (dx (x1 - x0)), 1 / (dy (x1 - x0)).  The spatial partners are the
// lanes g ^ XB (x) and g ^ YB (y) in every lane layout that calls it.
// s receives q's primitive variables.
template <class L, int ND, bool SOURCE = true>
GPR_D void dg_residual(const double *q, double *r, double sg, int i, int j, double hx, double hy,
                       const DevPar &P, Prim<L::THERMAL> &s) {
  constexpr int V = L::V;
  // lane bit layout: 1D g = 2t + i ; 2D g = 4t + 2i + j
  constexpr int XB = ND == 1 ? 1 : 2;  // flips i
  constexpr int YB = 1;                // flips j (2D)
  prim<L::THERMAL>(q, P, s);
  if (SOURCE) {
    source<L::THERMAL, V>(q, s, P, r, sg);
  } else {
#pragma unroll
    for (int k = 0; k < V; k++)
      r[k] = 0.0;
  }
#pragma unroll
  for (int d = 0; d < ND; d++) {
    const int lm = d == 0 ? XB : YB;
    const double c = sg * ((d == 0 ? i : j) ? -(d == 0 ? hx : hy) : (d == 0 ? hx : hy));
    // - B_d dq: columns other than d of the distortion, and the level sets
    const double vc[3] = {s.v[0] * c, s.v[1] * c, s.v[2] * c};
#pragma unroll
    for (int k = 5; k < V; k++) {
      const bool lset = k >= V - L::LSET;
      if (!lset && (k >= 14 || (k - 5) % 3 == d))
        continue;
      const double df = __shfl_xor_sync(0xffffffffu, q[k], lm) - q[k];
      r[k] = fma(-vc[d], df, r[k]);
      if (!lset) {
        const int col = (k - 5) % 3, dst = k - col + d;
        r[dst] = fma(vc[col], df, r[dst]);
      }
    }
    double F[V];
    flux_set<L::THERMAL, V>(q, s, d, P, F);
#pragma unroll
    for (int k = 0; k < V; k++)
      if (flux_support<L::THERMAL>(k, d))
        r[k] = fma(-c, __shfl_xor_sync(0xffffffffu, F[k], lm) - F[k], r[k]);
  }
}

template <class L, int ND, bool SOURCE = true>
GPR_D void dg_residual(const double *q, double *r, double sg, int i, int j, double hx, double hy,
                       const DevPar &P) {
  Prim<L::THERMAL> s;
  dg_residual<L, ND, SOURCE>(q, r, sg, i, j, hx, hy, P, s);
}

// The Picard map at this node, q_new(t, s) = sum_m DG_MATinv[t][m] (ENDVALS[0][m]
// W_s w + dt R(m, s)) / W_s = w + sum_m DG_MATinv[t][m] r_m: the initial
// condition's part is w itself (DG_MATinv maps ENDVALS[0] to 1).  r holds the
// residual at sg = dt W_t and is overwritten by q_new.
template <int V, int ND>
GPR_D void dg_solve_node(double *r, const double *w, int t, const Consts &C) {
  constexpr int TB = ND == 1 ? 2 : 4;  // flips t
  const double a = C.dgmatinv[t][t], b = C.dgmatinv[t][1 - t];
#pragma unroll
  for (int k = 0; k < V; k++)
    r[k] = fma(b, __shfl_xor_sync(0xffffffffu, r[k], TB), fma(a, r[k], w[k]));
}

// First Picard iteration.  From the standard initial guess q(t, s) = w(s)
// (initial_guess.cpp:4-15) the rhs at the two time nodes differs only by the
// weight W_t, so one thread per (cell, spatial node) evaluates it once (time
// weight 1) and writes q1 = w + DG_MATinv W r at both time nodes
// into qh; k_predictor_picard (first = 1) takes that as its first iterate
// and applies the reference's stopping test to it as usual.
template <class L, int ND, bool BATCH = false>
__global__ void __launch_bounds__(128) k_predictor_first(
    double *__restrict__ qh, const double *__restrict__ wh, long ncb,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double idx,
    double idy, DevPar Pv, Consts C, Batch B) {
  constexpr int V = L::V;
  constexpr int NS = ND == 1 ? NN : NN * NN;  // spatial nodes
  constexpr int NP = NN * NS;
  static_assert(NN == 2, "two time nodes");
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int g = threadIdx.x % NS;
  long c = gt / NS;
  bool valid = c < ncb;
  const long cc = valid ? c : 0;
  const int inst = BATCH ? B.inst_b[cc] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  if (BATCH) {
    dt = B.clk[5 * inst + 1];
    idx = B.idx[inst];
  }
  // the cells k_predictor_picard iterates (finished instances of a batch too);
  // a warp without one has nothing to write (800 x 400, two materials: 1.19
  // to 0.66 ms)
  const bool active = valid && (mask == nullptr || mask[c]);
  if (!__any_sync(0xffffffffu, active))
    return;
  const int i = ND == 1 ? g : g / NN, j = ND == 1 ? 0 : g % NN;
  double q[V], r[V];
  const double *wc = wh + (cc * NS + g) * V;
#pragma unroll
  for (int k = 0; k < V; k++)
    q[k] = valid ? wc[k] : 1.0;
  dg_residual<L, ND>(q, r, dt, i, j, idx * C.derv[0][1], idy * C.derv[0][1], P);
  if (!active)
    return;
  // q1_t = w + sum_m DG_MATinv[t][m] W_m r
  const double a0 = fma(C.dgmatinv[0][1], C.w[1], C.dgmatinv[0][0] * C.w[0]);
  const double a1 = fma(C.dgmatinv[1][1], C.w[1], C.dgmatinv[1][0] * C.w[0]);
  double *o0 = qh + (c * NP + g) * V, *o1 = qh + (c * NP + NS + g) * V;
#pragma unroll
  for (int k = 0; k < V; k++) {
    o0[k] = fma(a0, r[k], q[k]);
    o1[k] = fma(a1, r[k], q[k]);
  }
}

// Picard predictor.  ncb predictor cells; each warp holds 32/NP cells.
// status[c] (optional): GPR_PRED_PICARD | iterations << 8 when converged,
// GPR_PRED_FAILED when Picard did not converge (row left for the Newton pass,
// with the last Picard iterate written so the row is always defined).
struct PicardResume {
  int cap = 0;
  int *list = nullptr, *n = nullptr;
  int *it = nullptr;
  double *dmin = nullptr;
  const int *in = nullptr, *n_in = nullptr;
};

template <class L, int ND, bool BATCH = false>
__global__ void __launch_bounds__(128) k_predictor_picard(
    double *__restrict__ qh, const double *__restrict__ wh, long ncb,
    const uint8_t *__restrict__ mask, int32_t *__restrict__ status, double dt,
    const double *__restrict__ dt_dev, double idx, double idy, int stiff, DevPar Pv, Consts C,
    Batch B, int first, PicardResume R = PicardResume{}) {
  constexpr int V = L::V;
  constexpr int NS = ND == 1 ? NN : NN * NN;  // spatial nodes
  constexpr int NP = NN * NS;                 // space-time nodes
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int g = threadIdx.x % NP;
  long c = gt / NP;
  bool valid = c < ncb;
  if (R.in) {
    const long qi = gt / NP;
    valid = qi < *R.n_in;
    c = valid ? R.in[qi] : 0;
  }
  const int inst = BATCH ? B.inst_b[valid ? c : 0] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  if (BATCH) {
    dt = B.clk[5 * inst + 1];
    idx = B.idx[inst];
  }
  bool active = valid && (mask == nullptr || mask[c]);
  int t = g / NS, sidx = g % NS;
  int i = ND == 1 ? sidx : sidx / NN, j = ND == 1 ? 0 : sidx % NN;
  double w[V], q[V], qn[V];
  long cc = valid ? c : 0;
  const double *wc = wh + (cc * NS + sidx) * V;
  const double sg = dt * C.w[t], hx = idx * C.derv[0][1], hy = idy * C.derv[0][1];
  const float tolf = (float)C.dg_tol;
#pragma unroll
  for (int k = 0; k < V; k++) {
    w[k] = valid ? wc[k] : 1.0;
    q[k] = (R.in && valid) ? qh[(cc * NP + g) * V + k] : w[k];
  }
  // groups are aligned to NP lanes; the group shares the convergence decision
  unsigned lane = threadIdx.x & 31u;
  unsigned gmask = ((NP == 32) ? 0xffffffffu : ((1u << NP) - 1u)) << (lane & ~(NP - 1u));
  bool done = !active;
  int iters = 0;
  bool nan_seen = false;
  const int maxit = stiff ? 0 : C.dg_it;
  // Divergence detection: a cell whose largest update has grown DIVERGE
  // times above the smallest it reached is diverging and goes to the
  // stiff-source Newton pass at once instead of spending the rest of the
  // iteration cap; in a Newtonian fluid, whose iteration map is smooth, GROWN
  // times.  Measured with the oracle's iteration over 32 M cells (every
  // equation of state; Newtonian, power-law and Bingham fluids, elastoplastic
  // solids; V = 14, 15 and 17; tubes, 2D flows and batched instances, CFL 0.2 ..
  // 1), 20 M of them converging: a converging cell's updates grow by at most 10
  // times on the way, in a Newtonian fluid (8 M) 4 times, and no further in a
  // search that perturbs such cells towards larger growth.  Cells that fail
  // pass 32 times within 6 .. 20 iterations, 1e3 within 8 .. 25, or settle into
  // O(1) oscillations.
  // Those oscillations are told by their rate, in Newtonian fluids: r, the
  // largest update over its threshold, in windows of four iterations (their
  // maxima b after a); a cell whose r, continued at the rate (b / a) per window,
  // stands above 1e5 at the cap from two windows running goes to the Newton
  // pass too.  Converging cells: at most 10^1.6 in that measurement, 10^4.2 in
  // that search.  (One window tells too little: 10^3.2 and 10^7.4.  Nor does
  // the rate tell anything where the relaxation has a yield point or a steep
  // power: the iteration can leave a plateau from one update to the next, and
  // converging Bingham cells are predicted at 10^9 from one window and 10^7
  // from two.)  The windows begin at iteration 4 since with earlier or shorter
  // ones the transient's growth is taken for the rate.
  // Both are applied up to the reference's cap of 50, where they were measured:
  // eight iterations say nothing about the 300 of the differentiated forward,
  // where cells converge to 1e-13 after as many as 290.
  // The failing cells of a 256 x 256 vortex of viscosity 0.02 at CFL 0.8 stop
  // after 12 iterations, with the growth of 1e3 alone after 22, those of random
  // Newtonian flows after 11 instead of 17: 19.8 to 8.1 ms a step of that
  // vortex; one of 512 x 512, viscosity 0.01, at CFL 0.4, where every cell
  // converges, stays at 16.1 ms (r is taken from iteration 4 on only).
  const bool rated =
      maxit <= PICARD_RATE_CAP && !(P.flags & (GPR_SOLID | GPR_POWER_LAW | GPR_BINGHAM));
  const float grown = rated ? PICARD_GROWN : PICARD_DIVERGE;
  const bool resume = R.in != nullptr && valid;
  const int it0 = resume ? R.it[c] : 0;
  float dmin = resume ? (float)R.dmin[c] : F32_TOP;
  bool failed = false, deferred = false;
  float wa = 0.0f, wb = 0.0f;  // the last window's maximum and this one's
  bool hopeless = false;       // the last window's verdict
  for (int kq = 0;; kq++) {
    const int it = it0 + kq;
    // the same over the warp
    const bool late = (R.in != nullptr || kq >= PICARD_WINDOW0) && maxit <= PICARD_RATE_CAP;
    if (!done && it >= maxit) {
      failed = true;
      done = true;
    }
    if (!done && R.cap > 0 && kq == R.cap) {
      double *outd = qh + (c * NP + g) * V;
#pragma unroll
      for (int k = 0; k < V; k++)
        outd[k] = q[k];
      if (g == 0) {
        R.it[c] = it;
        R.dmin[c] = dmin;
        R.list[atomicAdd(R.n, 1)] = (int)c;
      }
      deferred = true;
      done = true;
    }
    if (__all_sync(0xffffffffu, done))
      break;
    // (a continuation never takes this branch, not even on its unused lanes,
    // whose it0 is 0: the other branch's shuffles need the whole warp)
    if (it == 0 && first && R.in == nullptr) {
      // the first iterate, from k_predictor_first
      const double *src = qh + (cc * NP + g) * V;
#pragma unroll
      for (int k = 0; k < V; k++)
        qn[k] = active ? src[k] : q[k];
    } else {
      dg_residual<L, ND>(q, qn, sg, i, j, hx, hy, P);
      dg_solve_node<V, ND>(qn, w, t, C);
    }
    // The reference's test |q1 - q0| > dg_tol (1 + |q0|) per entry.  Only the
    // difference needs FP64; an entry is decided in FP32 from the high words
    // (relative error of both sides below 3e-6) wherever the two sides differ
    // by more than 1e-5, and a cell that no entry so decides as changing takes
    // the FP64 test for the entries left open, so the decision is the FP64 one
    // (17 subtractions against 51 FP64 instructions).  The largest update,
    // which only the divergence test reads, is kept in FP32.
    bool big = false, open = false, hasnan = false;
    float dmax = 0.0f, rmax = 0.0f;
#pragma unroll
    for (int k = 0; k < V; k++) {
      const float df = f32_abs_hi(qn[k] - q[k]), qf = f32_abs_hi(q[k]);
      const float th = fmaf(tolf, qf, tolf);
      if (late)
        rmax = fmaxf(rmax, __fdividef(df, th));
      const bool ok = fmaxf(df, qf) < F32_TOP;
      big = big || (ok && df > th * 1.00001f);
      open = open || !ok || df > th * 0.99999f;
      dmax = fmaxf(dmax, df);
    }
    unsigned bigm = __ballot_sync(0xffffffffu, big) & gmask;
    if (open && !bigm) {
#pragma unroll
      for (int k = 0; k < V; k++) {
        if (fabs(qn[k] - q[k]) > C.dg_tol * (1.0 + fabs(q[k])))
          big = true;
        if (fp_abs_bits(qn[k]) > FP_INF_BITS)
          hasnan = true;
      }
    }
    bigm = __ballot_sync(0xffffffffu, big) & gmask;
    const unsigned nanm = __ballot_sync(0xffffffffu, hasnan) & gmask;
#pragma unroll
    for (int o = 1; o < NP; o <<= 1)
      dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if (!done && bigm && it >= 3 && dmax > grown * dmin) {
      nan_seen = true;  // hand over to the Newton pass
      done = true;
      iters = it + 1;
    }
    if (late) {
#pragma unroll
      for (int o = 1; o < NP; o <<= 1)
        rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
      if (it >= PICARD_WINDOW0) {
        wb = fmaxf(wb, rmax);
        if ((it - PICARD_WINDOW0) % 4 == 3) {
          const float lb = __log2f(wb);
          const float lp = lb + 0.25f * (float)(maxit - 1 - it) * (lb - __log2f(wa));
          const bool above = it >= PICARD_WINDOW0 + 7 && lp > PICARD_HOPELESS;
          if (!done && bigm && rated && above && hopeless) {
            nan_seen = true;  // hand over to the Newton pass
            done = true;
            iters = it + 1;
          }
          hopeless = above;
          wa = wb;
          wb = 0.0f;
        }
      }
    }
    if (!done)
      dmin = fminf(dmin, dmax);
    if (!done) {
      iters = it + 1;
      if (bigm) {
#pragma unroll
        for (int k = 0; k < V; k++)
          q[k] = qn[k];
      } else if (nanm) {
        nan_seen = true;
        done = true;
      } else {
#pragma unroll
        for (int k = 0; k < V; k++)
          q[k] = qn[k];
        done = true;
        if (active) {
          double *out = qh + (c * NP + g) * V;
#pragma unroll
          for (int k = 0; k < V; k++)
            out[k] = q[k];
          if (status && g == 0)
            status[c] = GPR_PRED_PICARD | (iters << 8);
        }
      }
    }
  }
  if (active && !deferred && (failed || nan_seen)) {
    // Picard failed: write the initial guess and flag the cell for the
    // stiff-source Newton pass with a NaN in its first entry
    double *out = qh + (c * NP + g) * V;
#pragma unroll
    for (int k = 0; k < V; k++)
      out[k] = w[k];
    if (g == 0)
      out[0] = __longlong_as_double(0x7ff8000000000bad);
    if (status && g == 0)
      status[c] = GPR_PRED_FAILED | (iters << 8);
  }
  if (valid && !active && status && g == 0)
    status[c] = GPR_PRED_PICARD;
}

// ---------------------------------------------------------------------------
// midstepper (split/homogeneous.cpp:5-67): the half step of the homogeneous
// system at the WENO nodes before the split scheme's FV update,
//   w_s -= dt/2 ((dF/dx + B_x dw/dx) / dx [+ (dG/dy + B_y dw/dy) / dy]),
// derivatives by DERVALS within the cell.  One thread per spatial node, the
// cell's NS = N^d lanes adjacent (x partner lane ^ (ND == 1 ? 1 : 2), y
// partner lane ^ 1).
template <class L, int ND>
__global__ void __launch_bounds__(128) k_midstep(double *__restrict__ wh, long ncb,
                                                 const uint8_t *__restrict__ mask, double dt,
                                                 const double *__restrict__ dt_dev, double idx,
                                                 double idy, DevPar P, Consts C) {
  constexpr int V = L::V;
  constexpr int NS = ND == 1 ? NN : NN * NN;
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int g = threadIdx.x % NS;
  const long c = gt / NS;
  const bool valid = c < ncb;
  const long cc = valid ? c : 0;
  const bool active = valid && (mask == nullptr || mask[cc]);
  const int a = ND == 1 ? g : g / NN, b = ND == 1 ? 0 : g % NN;
  double w[V], r[V];
  double *wc = wh + (cc * NS + g) * V;
#pragma unroll
  for (int k = 0; k < V; k++)
    w[k] = wc[k];
  dg_residual<L, ND, false>(w, r, 0.5 * dt, a, b, idx * C.derv[0][1], idy * C.derv[0][1], P);
  if (active) {
#pragma unroll
    for (int k = 0; k < V; k++)
      wc[k] = w[k] + r[k];
  }
}

// ---------------------------------------------------------------------------
// Stiff-source Newton pass for the cells whose Picard iteration failed (the
// reference leaves their rows unwritten, dg1.cpp:91-110, or falls back to a
// Jacobian-free Newton-Krylov solve on NaN, dg1.cpp:100-105).
//
// Iteration on the predictor fixed point Fp(q) = DG_U q - Ww - dt R(q) = 0:
//   delta = (DG_U - dt W dS/dq)^-1 (Ww + dt R(q) - DG_U q),   q += delta,
// with dS/dq the exact local Jacobian of the relaxation sources at each
// space-time node (distortion 9x9, heat flux 3x3): implicit in the stiff
// sources, explicit in the fluxes; with dS/dq = 0 it is the Picard update.
// Per spatial node the correction couples the N = 2 time nodes through
// DG_MAT: an 18x18 system for A and a 6x6 system for rho J, assembled in
// shared memory by the node's two lanes and solved by one lane each
// (partial pivoting); the other variables use DG_MAT^-1 directly.

template <bool TH>
GPR_D void stiff_jacobian_rows(const double *q, const Prim<TH> &s, const DevPar &P, double a,
                               double mdiag, float *rowsA, int ldA, float *rowsJ, int ldJ) {
  // rowsA[i*ldA + j] (i = 0..8, j = 0..8): M[t][t] delta_ij - a JA[i][j]
  const double *A = q + 5;
  double H[9], dG[9];
  double G00 = A[0] * A[0] + A[3] * A[3] + A[6] * A[6];
  double G11 = A[1] * A[1] + A[4] * A[4] + A[7] * A[7];
  double G22 = A[2] * A[2] + A[5] * A[5] + A[8] * A[8];
  double G01 = A[0] * A[1] + A[3] * A[4] + A[6] * A[7];
  double G02 = A[0] * A[2] + A[3] * A[5] + A[6] * A[8];
  double G12 = A[1] * A[2] + A[4] * A[5] + A[7] * A[8];
  double t3 = (G00 + G11 + G22) * (1.0 / 3.0);
  dG[0] = G00 - t3; dG[1] = G01; dG[2] = G02;
  dG[3] = G01; dG[4] = G11 - t3; dG[5] = G12;
  dG[6] = G02; dG[7] = G12; dG[8] = G22 - t3;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int m = 0; m < 3; m++)
      H[3 * i + m] = A[3 * i] * A[3 * m] + A[3 * i + 1] * A[3 * m + 1] + A[3 * i + 2] * A[3 * m + 2];
  double dA = det3(A);
  int newtonian = !(P.flags & (GPR_SOLID | GPR_POWER_LAW | GPR_BINGHAM));
  double th = theta1inv<TH>(q, s, P);
  double id = rcp64(dA);
  double Ai[9];  // A^-1
  Ai[0] = (A[4] * A[8] - A[5] * A[7]) * id;
  Ai[1] = (A[2] * A[7] - A[1] * A[8]) * id;
  Ai[2] = (A[1] * A[5] - A[2] * A[4]) * id;
  Ai[3] = (A[5] * A[6] - A[3] * A[8]) * id;
  Ai[4] = (A[0] * A[8] - A[2] * A[6]) * id;
  Ai[5] = (A[2] * A[3] - A[0] * A[5]) * id;
  Ai[6] = (A[3] * A[7] - A[4] * A[6]) * id;
  Ai[7] = (A[1] * A[6] - A[0] * A[7]) * id;
  Ai[8] = (A[0] * A[4] - A[1] * A[3]) * id;
  double fth = newtonian ? (5.0 / 3.0) * th : 0.0;
  double ca = a * s.cs2;  // a (-JA) = ca (th v + AdG dth)
  // The 81 entries in FP32: the rows are stored in FP32 for the FP32
  // correction solve (the residual stays FP64, so the converged point is the
  // FP64 fixed point), and FP32 runs beside the FP64 pipe at full rate.
  float Af[9], dGf[9], Hf[9], Aif[9], AdGf[9];
#pragma unroll
  for (int k = 0; k < 9; k++) {
    Af[k] = (float)A[k];
    dGf[k] = (float)dG[k];
    Hf[k] = (float)H[k];
    Aif[k] = (float)(Ai[k] * fth);
    AdGf[k] = (float)(s.AdG[k] * ca);
  }
  const float cth = (float)(ca * th), md = (float)mdiag;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      int rr = 3 * i + j;
#pragma unroll
      for (int m = 0; m < 3; m++)
#pragma unroll
        for (int n = 0; n < 3; n++) {
          float v = (i == m ? dGf[3 * n + j] : 0.0f) + Af[3 * i + n] * Af[3 * m + j] +
                    (n == j ? Hf[3 * i + m] : 0.0f) -
                    (2.0f / 3.0f) * Af[3 * i + j] * Af[3 * m + n];
          float e = cth * v + AdGf[rr] * Aif[3 * n + m];
          rowsA[rr * ldA + 3 * m + n] = (rr == 3 * m + n ? md : 0.0f) + e;
        }
    }
  if (TH) {
    double f = a * P.calpha2 * P.ikappa;  // -a JJ = f (T/rho I + J dT)
#pragma unroll
    for (int l = 0; l < 3; l++)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double dT = -P.calpha2 * s.J[k] * s.ir * P.icv;
        rowsJ[l * ldJ + k] =
            (float)((l == k ? mdiag : 0.0) + f * ((l == k ? s.T * s.ir : 0.0) + s.J[l] * dT));
      }
  }
}

// In-place Gaussian elimination with partial pivoting on the n x n system
// M (leading dimension ld) with right-hand side b; solution left in b.  The
// stiff pass solves its correction systems in FP32: the residual is FP64, so
// the converged fixed point is the FP64 one and the single-precision
// Jacobian only changes the (already linear) contraction rate slightly.
template <int n, class R>
GPR_D bool smem_solve(R *M, int ld, R *b) {
  for (int c = 0; c < n; c++) {
    int p = c;
    R best = fabs(M[c * ld + c]);
#pragma unroll 4
    for (int r = c + 1; r < n; r++) {
      R v = fabs(M[r * ld + c]);
      if (v > best) {
        best = v;
        p = r;
      }
    }
    if (!(best > R(0)))
      return false;
    if (p != c) {
#pragma unroll 4
      for (int j = c; j < n; j++) {
        R tmp = M[c * ld + j];
        M[c * ld + j] = M[p * ld + j];
        M[p * ld + j] = tmp;
      }
      R tmp = b[c];
      b[c] = b[p];
      b[p] = tmp;
    }
    R inv = R(1) / M[c * ld + c];
    for (int r = c + 1; r < n; r++) {
      R f = M[r * ld + c] * inv;
#pragma unroll 4
      for (int j = c + 1; j < n; j++)
        M[r * ld + j] -= f * M[c * ld + j];
      b[r] -= f * b[c];
    }
  }
  for (int r = n - 1; r >= 0; r--) {
    R acc = b[r];
#pragma unroll 4
    for (int j = r + 1; j < n; j++)
      acc -= M[r * ld + j] * b[j];
    b[r] = acc / M[r * ld + r];
  }
  return true;
}

template <class L, int ND> struct StiffSmem {
  static constexpr int NS = ND == 1 ? NN : NN * NN;
  static constexpr int NA = 9 * NN, NJ = 3 * NN;
  // odd number of floats: the solver lanes of neighbouring spatial nodes
  // then start on different shared-memory banks
  static constexpr int raw = NA * NA + NA + (L::THERMAL ? NJ * NJ + NJ : 0);
  static constexpr int per_node = raw | 1;
  static constexpr int CPB = 8;  // cells per 64-thread block (2D: 8 lanes each)
  static constexpr int per_cell = NS * per_node;
};

template <class L, int ND, bool BATCH = false>
__global__ void __launch_bounds__(64) k_predictor_stiff(
    double *__restrict__ qh, const double *__restrict__ wh, long ncb,
    const uint8_t *__restrict__ mask, int32_t *__restrict__ status, double dt_in,
    const double *__restrict__ dt_dev, double idx_in, double idy, DevPar Pv, Consts C,
    Batch B) {
  constexpr int V = L::V;
  constexpr int NS = ND == 1 ? NN : NN * NN;
  constexpr int NP = NN * NS;
  constexpr int TB = ND == 1 ? 2 : 4;  // flips t
  constexpr int NA = 9 * NN, NJ = 3 * NN;
  using SM = StiffSmem<L, ND>;
  extern __shared__ float fsmem[];
  if (dt_dev)
    dt_in = *dt_dev;
  const int g = threadIdx.x % NP;
  const int t = g / NS, sidx = g % NS;
  const int i = ND == 1 ? sidx : sidx / NN, j = ND == 1 ? 0 : sidx % NN;
  float *cellmem = fsmem + (threadIdx.x / NP) * SM::per_cell;
  float *Am = cellmem + sidx * SM::per_node;  // 18 x 18
  float *Ab = Am + NA * NA;                   // 18
  float *Jm = Ab + NA;                        // 6 x 6
  float *Jb = Jm + NJ * NJ;                   // 6
  const unsigned lane = threadIdx.x & 31u;
  const unsigned gmask = ((NP == 32) ? 0xffffffffu : ((1u << NP) - 1u)) << (lane & ~(NP - 1u));
  const double f = C.endv[0][t];
  const double M0 = C.dgmat[t][t], M1 = C.dgmat[t][1 - t];
  const float tolf = (float)C.stiff_tol;
  const long cells_per_block = blockDim.x / NP;
  // persistent: blocks stride over the cells; the loop bound is uniform in
  // the block so every lane takes part in the warp-level exchanges
  for (long base = blockIdx.x * cells_per_block; base < ncb;
       base += (long)gridDim.x * cells_per_block) {
    long c = base + threadIdx.x / NP;
    bool valid = c < ncb;
    long cc = valid ? c : 0;
    bool active = valid && (mask == nullptr || mask[cc]);
    double flag = active ? qh[cc * NP * V] : 0.0;  // NaN sentinel of the Picard pass
    active = active && (flag != flag);
    if (__all_sync(0xffffffffu, !active))
      continue;
    const int inst = BATCH ? B.inst_b[cc] : 0;
    const DevPar &P = BATCH ? B.P[inst] : Pv;
    const double dt = BATCH ? B.clk[5 * inst + 1] : dt_in;
    const double idx = BATCH ? B.idx[inst] : idx_in;
    const double a_t = dt * C.w[t];
    const double hx = idx * C.derv[0][1], hy = idy * C.derv[0][1];
    double fw[V], q[V], r[V], other[V];
    const double *wc = wh + (cc * NS + sidx) * V;
#pragma unroll
    for (int k = 0; k < V; k++) {
      double w = active ? wc[k] : 1.0;
      fw[k] = f * w;
      q[k] = w;
    }
    bool done = !active;
    bool ok = false;
    int iters = 0;
    for (int it = 0; it < C.stiff_it; it++) {
      if (__all_sync(0xffffffffu, done))
        break;
      Prim<L::THERMAL> st;
      dg_residual<L, ND>(q, r, a_t, i, j, hx, hy, P, st);
      // the fixed point's residual over W_s: r + ENDVALS[0][t] w - sum_m
      // DG_MAT[t][m] q(m)
      shfl_vec<V>(q, other, TB);
#pragma unroll
      for (int k = 0; k < V; k++)
        r[k] += fma(-M1, other[k], fma(-M0, q[k], fw[k]));
      if (!done) {
        // this time node's diagonal block A_t = M_tt I - a_t dS/dA of the
        // 18 x 18 Newton matrix (the off-diagonal blocks are M_t,1-t I) and
        // its right-hand side
        stiff_jacobian_rows<L::THERMAL>(q, st, P, a_t, M0, Am + t * 9 * NA + t * 9, NA,
                                        Jm + t * 3 * NJ + t * 3, NJ);
#pragma unroll
        for (int a = 0; a < 9; a++)
          Ab[t * 9 + a] = (float)r[5 + a];
        if (L::THERMAL) {
#pragma unroll
          for (int a = 0; a < 3; a++)
            Jb[t * 3 + a] = (float)r[14 + a];
        }
      }
      __syncwarp();
      // Block elimination of [[A0, m01 I], [m10 I, A1]] [x0; x1] = [b0; b1]:
      // (A0 A1 - m01 m10 I) x1 = A0 b1 - m10 b0 and x0 = (b1 - A1 x1) / m10,
      // a 9 x 9 solve (3 x 3 for the heat flux) in place of 18 x 18 (6 x 6).
      // The two time-node lanes form the reduced matrix's rows (into block
      // (0, 1) of Am), lane t = 0 its right-hand side (block (1, 0)'s first
      // row) and lane t = 1 the heat-flux system.
      const float m01 = (float)C.dgmat[0][1], m10 = (float)C.dgmat[1][0];
      const float *A0 = Am, *A1 = Am + 9 * NA + 9;
      float *Rm = Am + 9, *Rb = Am + 9 * NA;
      const float *J0 = Jm, *J1 = Jm + 3 * NJ + 3;
      float *RJm = Jm + 3, *RJb = Jm + 3 * NJ;
      if (!done) {
        const int r0 = t == 0 ? 0 : 5, r1 = t == 0 ? 5 : 9;
        for (int rr = r0; rr < r1; rr++) {
#pragma unroll
          for (int c = 0; c < 9; c++) {
            float acc = rr == c ? -m01 * m10 : 0.0f;
#pragma unroll
            for (int k = 0; k < 9; k++)
              acc = fmaf(A0[rr * NA + k], A1[k * NA + c], acc);
            Rm[rr * NA + c] = acc;
          }
        }
        if (t == 0) {
#pragma unroll
          for (int rr = 0; rr < 9; rr++) {
            float acc = -m10 * Ab[rr];
#pragma unroll
            for (int k = 0; k < 9; k++)
              acc = fmaf(A0[rr * NA + k], Ab[9 + k], acc);
            Rb[rr] = acc;
          }
        } else if (L::THERMAL) {
#pragma unroll
          for (int rr = 0; rr < 3; rr++) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
              float acc = rr == c ? -m01 * m10 : 0.0f;
#pragma unroll
              for (int k = 0; k < 3; k++)
                acc = fmaf(J0[rr * NJ + k], J1[k * NJ + c], acc);
              RJm[rr * NJ + c] = acc;
            }
            float acc = -m10 * Jb[rr];
#pragma unroll
            for (int k = 0; k < 3; k++)
              acc = fmaf(J0[rr * NJ + k], Jb[3 + k], acc);
            RJb[rr] = acc;
          }
        }
      }
      __syncwarp();
      bool solved = true;
      if (!done) {
        if (t == 0)
          solved = smem_solve<9>(Rm, NA, Rb);
        else if (L::THERMAL)
          solved = smem_solve<3>(RJm, NJ, RJb);
      }
      __syncwarp();
      // non-stiff variables: DG_MAT^-1 g (partner time node's residual)
      shfl_vec<V>(r, other, TB);
      double delta[V];
      const double ia = C.dgmatinv[t][t], ib = C.dgmatinv[t][1 - t];
#pragma unroll
      for (int k = 0; k < V; k++)
        delta[k] = ia * r[k] + ib * other[k];
      // stiff variables: x1 from the reduced solve, x0 = (b1 - A1 x1) / m10
      const float im10 = 1.0f / m10;
#pragma unroll
      for (int a = 0; a < 9; a++) {
        float x = Rb[a];
        if (t == 0) {
          float acc = Ab[9 + a];
#pragma unroll
          for (int k = 0; k < 9; k++)
            acc = fmaf(-A1[a * NA + k], Rb[k], acc);
          x = acc * im10;
        }
        delta[5 + a] = (double)x;
      }
      if (L::THERMAL) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
          float x = RJb[a];
          if (t == 0) {
            float acc = Jb[3 + a];
#pragma unroll
            for (int k = 0; k < 3; k++)
              acc = fmaf(-J1[a * NJ + k], RJb[k], acc);
            x = acc * im10;
          }
          delta[14 + a] = (double)x;
        }
      }
      __syncwarp();
      // |delta| > stiff_tol (1 + |qn|), in FP32 from the high words wherever the
      // sides differ by more than 1e-5, as the Picard pass's test
      bool big = false, open = false, bad = !solved;
#pragma unroll
      for (int k = 0; k < V; k++) {
        const double qn = q[k] + delta[k];
        const float df = f32_abs_hi(delta[k]), qf = f32_abs_hi(qn);
        const float th = fmaf(tolf, qf, tolf);
        const bool in = fmaxf(df, qf) < F32_TOP;
        big = big || (in && df > th * 1.00001f);
        open = open || !in || df > th * 0.99999f;
        if (!done)
          q[k] = qn;
      }
      unsigned bigm = __ballot_sync(0xffffffffu, big) & gmask;
      if (open) {
#pragma unroll
        for (int k = 0; k < V; k++) {
          const double qn = done ? q[k] + delta[k] : q[k];
          if (!bigm && fabs(delta[k]) > C.stiff_tol * (1.0 + fabs(qn)))
            big = true;
          if (fp_abs_bits(qn) > FP_INF_BITS)
            bad = true;
        }
      }
      bigm = __ballot_sync(0xffffffffu, big) & gmask;
      unsigned badm = __ballot_sync(0xffffffffu, bad) & gmask;
      if (!done) {
        iters = it + 1;
        if (badm) {
          done = true;
        } else if (!bigm) {
          done = true;
          ok = true;
        }
      }
    }
    if (active) {
      double *out = qh + (cc * NP + g) * V;
#pragma unroll
      for (int k = 0; k < V; k++)
        out[k] = q[k];
      if (status && g == 0)
        status[cc] = (ok ? GPR_PRED_NEWTON : GPR_PRED_FAILED) | (iters << 8);
    }
  }
}

// ---------------------------------------------------------------------------
// Finite-volume update (solvers/fv/fv.cpp:11-297).
//
// Face pass: one thread per (face, time node t[, transverse node s]).  It
// extrapolates qL, qR to the face, evaluates the Rusanov dissipation
// D = max(lambda_L, lambda_R)(qL - qR) + F(qL) + F(qR) (fluxes.cpp:66-75) and
// the path integral Bint (fluxes.cpp:9-20), weights them, and the NQ lanes
// of a face reduce with shuffles.  Face results: fb[face][0][k] (to the left
// cell, subtracted) and fb[face][1][k] (to the right cell).

// Bint = sum_n W_n B_d(qL + x_n dq) dq, dq = qR - qL (fluxes.cpp:9-20).  B_d
// is linear in the velocity and needs nothing else of the state, so the path
// nodes' velocities are averaged first and one product taken; b is written on
// the rows where it can be nonzero and zeroed elsewhere.
template <class L, int NQ>
GPR_D void path_product(const double *ql, const double *dq, int d, const double *nodes,
                        const double *wts, double *b) {
  double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int n = 0; n < NQ; n++) {
    const double wr = wts[n] * rcp64(fma(nodes[n], dq[0], ql[0]));
#pragma unroll
    for (int c = 0; c < 3; c++)
      v[c] = fma(wr, fma(nodes[n], dq[2 + c], ql[2 + c]), v[c]);
  }
  bdot<L::V, L::LSET>(v, dq, d, b);
}

// Rusanov interface terms at one point: f = D + F(qL) + F(qR) and b = Bint.
template <class L, int NQ>
GPR_D void rusanov_point(const double *ql, const double *qr, int d, const DevPar &P,
                         const double *nodes, const double *wts, double *f, double *b) {
  constexpr int V = L::V;
  Prim<L::THERMAL> sl, sr;
  prim<L::THERMAL>(ql, P, sl);
  prim<L::THERMAL>(qr, P, sr);
  const double m1 = max_abs_eigs<L::THERMAL>(ql, sl, d, P);
  const double m2 = max_abs_eigs<L::THERMAL>(qr, sr, d, P);
  const double m = m1 > m2 ? m1 : m2;  // std::max(m1, m2)
  double fl[V], dq[V];
  flux_set<L::THERMAL, V>(ql, sl, d, P, fl);
  flux_set<L::THERMAL, V>(qr, sr, d, P, f);
#pragma unroll
  for (int k = 0; k < V; k++) {
    dq[k] = qr[k] - ql[k];
    f[k] = flux_support<L::THERMAL>(k, d) ? fma(-m, dq[k], fl[k] + f[k]) : -m * dq[k];
  }
  path_product<L, NQ>(ql, dq, d, nodes, wts, b);
}

template <class L>
GPR_D void interface_point(const double *ql, const double *qr, int d, const DevPar &P,
                           const Consts &C, double *f, double *b) {
  rusanov_point<L, NN>(ql, qr, d, P, C.nodes, C.w, f, b);
}

// 1D faces i = 0..nx between predictor cells i and i+1.  NQ = N lanes per
// face (time nodes).
template <class L, bool BATCH = false>
__global__ void __launch_bounds__(128) k_faces1d(
    double *__restrict__ fb, const double *__restrict__ qh, long nface,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double idx,
    int time_dg, DevPar Pv, Consts C, Batch B) {
  constexpr int V = L::V;
  constexpr int NQ = NN;
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int t = threadIdx.x % NQ;
  long face = gt / NQ;
  bool valid = face < nface;
  long fo = valid ? face : 0;
  // predictor cell on the left of the face (packed index in the batched form)
  long fi = fo;
  const int inst = BATCH ? B.inst_f[fo] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  if (BATCH) {
    fi = B.off_b[inst] + (fo - B.off_f[inst]);
    dt = B.clk[5 * inst + 1];
    idx = B.idx[inst];
  }
  bool active = valid && (mask == nullptr || (mask[fi] && mask[fi + 1])) && (time_dg || t == 0);
  int nt = time_dg ? NN : 1;
  double ql[V], qr[V], f[V], b[V];
  const double *ql_ = qh + (fi * nt + (time_dg ? t : 0)) * NN * V;
  const double *qr_ = qh + ((fi + 1) * nt + (time_dg ? t : 0)) * NN * V;
#pragma unroll
  for (int k = 0; k < V; k++) {
    ql[k] = C.endv[1][0] * ql_[k] + C.endv[1][1] * ql_[V + k];
    qr[k] = C.endv[0][0] * qr_[k] + C.endv[0][1] * qr_[V + k];
  }
  const double kk = dt * idx * (time_dg ? 0.5 * GAUSS_W : 0.5);
  if (active) {
    interface_point<L>(ql, qr, 0, P, C, f, b);
  } else {
#pragma unroll
    for (int k = 0; k < V; k++)
      f[k] = b[k] = 0.0;
  }
  face_reduce_store<V, NN>(b, f, kk, active, valid, t, fb + fo * 2 * V);
}

// 1D faces for small grids, where a kernel's time is the length of one
// lane's FP64 instruction chain: one lane per (face, time node, side).  The
// lane of side 0 (1) evaluates the primitives, wave speed and flux of qL
// (qR) and the path integral's node 0 (1); the wave speeds are exchanged,
// the side-0 lane adds the dissipation, and the four lanes' contributions
// are summed by the reduce-scatter (the same terms as interface_point).
template <class L, bool BATCH>
GPR_D void faces1d_split_body(double *__restrict__ fb, const double *__restrict__ qh,
                              long nface, const uint8_t *__restrict__ mask, double dt,
                              double idx, int time_dg, const DevPar &Pv, const Consts &C,
                              const Batch &B, long face, int lq, bool inrange, long fbase) {
  constexpr int V = L::V;
  static_assert(NN == 2, "two time nodes and two path nodes");
  const int t = lq >> 1, side = lq & 1;
  bool valid = inrange && face < nface;
  const long fo = valid ? face : 0;
  // predictor cell on the left of the face (packed index in the batched form)
  long fi = fo;
  const int inst = BATCH ? B.inst_f[fo] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  if (BATCH) {
    fi = B.off_b[inst] + (fo - B.off_f[inst]);
    dt = B.clk[5 * inst + 1];
    idx = B.idx[inst];
  }
  bool active = valid && (mask == nullptr || (mask[fi] && mask[fi + 1])) && (time_dg || t == 0);
  int nt = time_dg ? NN : 1;
  // each lane extrapolates its own side and takes the other from its partner
  double qs[V], ql[V], f[V], b[V], dq[V];
  const double *qs_ = qh + ((fi + side) * nt + (time_dg ? t : 0)) * NN * V;
  const double e0 = C.endv[1 - side][0], e1 = C.endv[1 - side][1];
#pragma unroll
  for (int k = 0; k < V; k++) {
    qs[k] = e0 * qs_[k] + e1 * qs_[V + k];
    const double o = __shfl_xor_sync(0xffffffffu, qs[k], 1);
    ql[k] = side ? o : qs[k];
    dq[k] = (side ? qs[k] : o) - ql[k];
  }
  const double kk = dt * idx * (time_dg ? 0.5 * GAUSS_W : 0.5);
  Prim<L::THERMAL> ps;
  prim<L::THERMAL>(qs, P, ps);
  const double lam = max_abs_eigs<L::THERMAL>(qs, ps, 0, P);
  const double lo = __shfl_xor_sync(0xffffffffu, lam, 1);
  const double m1 = side ? lo : lam, m2 = side ? lam : lo;  // lambda(qL), lambda(qR)
  const double m = m1 > m2 ? m1 : m2;                        // std::max(m1, m2)
  flux_set<L::THERMAL, V>(qs, ps, 0, P, f);
  // the dissipation -m dq once per point (side 0)
  const double ms = side == 0 ? -m : 0.0;
#pragma unroll
  for (int k = 0; k < V; k++)
    f[k] = flux_support<L::THERMAL>(k, 0) ? fma(ms, dq[k], f[k]) : ms * dq[k];
  // Bint node `side`: W_n B(qL + x_n dq) dq   (fluxes.cpp:9-20)
  {
    const double xn = C.nodes[side];
    const double wr = GAUSS_W * rcp64(fma(xn, dq[0], ql[0]));
    const double v[3] = {fma(xn, dq[2], ql[2]) * wr, fma(xn, dq[3], ql[3]) * wr,
                         fma(xn, dq[4], ql[4]) * wr};
    bdot<V, L::LSET>(v, dq, 0, b);
  }
  face_reduce_store<V, 4>(b, f, kk, active, valid, lq, fb + (fo - fbase) * 2 * V);
}

template <class L, bool BATCH = false>
__global__ void __launch_bounds__(128) k_faces1d_split(
    double *__restrict__ fb, const double *__restrict__ qh, long nface,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double idx,
    int time_dg, DevPar Pv, Consts C, Batch B) {
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  faces1d_split_body<L, BATCH>(fb, qh, nface, mask, dt, idx, time_dg, Pv, C, B, gt / 4,
                               threadIdx.x % 4, true, 0);
}

// 2D faces: direction DIR (compile-time: a run-time axis makes the
// kernel keep 1.3 KB of its state in local memory), faces (i, j) of the (nx+1) x (ny+1) face grid,
// between predictor cells (i, j) and (i+1, j) (DIR 0) or (i, j+1) (DIR 1);
// ih = 1 / dx_DIR; NQ = N*N lanes per face (time node t, transverse node s).  parity < 0:
// every face, contributions written to fb[face][2][V] (the face-flux
// entry points); parity 0 / 1: the faces of that parity along DIR, applied
// to u (passed as fb) in place, the conservative update of interfs2.
// point(ql, qr) evaluates f and b at one quadrature point.
template <class L, int DIR, class Point>
GPR_D void faces2d_body(double *__restrict__ fb, const double *__restrict__ qh, int nx, int ny,
                        const uint8_t *__restrict__ mask, double dt,
                        const double *__restrict__ dt_dev, double ih, int time_dg,
                        const Consts &C, int parity, double (&f)[L::V], double (&b)[L::V],
                        Point point) {
  constexpr int V = L::V;
  constexpr int NQ = NN * NN;
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int lq = threadIdx.x % NQ;
  int t = lq / NN, s = lq % NN;
  const Face2 F = face2_of(gt / NQ, nx, ny, DIR, parity);
  const bool valid = F.valid;
  const long fi = F.fi;
  const int i = F.i, j = F.j;
  long cb = (long)i * (ny + 2) + j;
  long cn = DIR == 0 ? cb + (ny + 2) : cb + 1;
  bool geo = DIR == 0 ? (j > 0) : (i > 0);
  const bool face_on = valid && geo && (mask == nullptr || (mask[cb] && mask[cn]));
  bool active = face_on && (time_dg || t == 0);
  // in place, a warp of faces that are off has nothing to apply (800 x 400,
  // two materials: 3.12 to 2.73 ms)
  if (parity >= 0 && !__any_sync(0xffffffffu, face_on))
    return;
  int nt = time_dg ? NN : 1;
  int tt = time_dg ? t : 0;
  const double *q0 = qh + (cb * nt + tt) * NN * NN * V;
  const double *q1 = qh + (cn * nt + tt) * NN * NN * V;
  double ql[V], qr[V];
  // endpts2d (evaluations.cpp:20-35): DIR 0 -> nodes (m, s); DIR 1 -> (s, m)
  long o0 = DIR == 0 ? (long)s * V : (long)s * NN * V;
  long st = DIR == 0 ? (long)NN * V : (long)V;
#pragma unroll
  for (int k = 0; k < V; k++) {
    ql[k] = C.endv[1][0] * q0[o0 + k] + C.endv[1][1] * q0[o0 + st + k];
    qr[k] = C.endv[0][0] * q1[o0 + k] + C.endv[0][1] * q1[o0 + st + k];
  }
  // W_t W_s dt / (2 h)
  const double kk = dt * ih * (time_dg ? 0.5 * GAUSS_W * GAUSS_W : 0.5 * GAUSS_W);
  if (active) {
    point(ql, qr);
  } else {
#pragma unroll
    for (int k = 0; k < V; k++)
      f[k] = b[k] = 0.0;
  }
  if (parity < 0) {
    face_reduce_store<V, NQ>(b, f, kk, active, valid, lq, fb + fi * 2 * V);
  } else {
    double *uL, *uR;
    face2_cells(fb, i, j, nx, ny, DIR, V, uL, uR);
    face_reduce_apply<V, NQ>(b, f, kk, active, face_on, lq, uL, uR);
  }
}

template <class L, int DIR>
__global__ void __launch_bounds__(128) k_faces2d(
    double *__restrict__ fb, const double *__restrict__ qh, int nx, int ny,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double ih,
    int time_dg, DevPar P, Consts C, int parity = -1) {
  double f[L::V], b[L::V];
  faces2d_body<L, DIR>(fb, qh, nx, ny, mask, dt, dt_dev, ih, time_dg, C, parity, f, b,
                       [&](const double *ql, const double *qr) {
                         interface_point<L>(ql, qr, DIR, P, C, f, b);
                       });
}

// Parts of the FV update k_cells applies: the volume term (centers1 /
// centers2, fv.cpp:11-109) and the face contributions (interfs1 / interfs2,
// fv.cpp:111-279); fv_launcher applies both.
constexpr int FV_CENTERS = 1, FV_INTERFS = 2, FV_BOTH = 3;

// Cell pass: one thread per (cell, space-time node): the volume term
// w_t w_s (S - B dq/dx [- B dq/dy]) (fv.cpp:11-109), reduced over the cell's
// NP lanes, then u += volume - face contributions (the parts selected).  hx,
// hy: 1 / (dx (x1 - x0)), 1 / (dy (x1 - x0)), as in dg_residual.
// The body for cell c (u index), lane g of its NP lanes; fbx[(fo - fbase)]
// holds the 1D face on the cell's left (fbase: the first face of a tile
// staged in shared memory, else 0).
template <class L, int ND, bool BATCH>
GPR_D void cells_body(double *__restrict__ u, const double *__restrict__ qh,
                      const double *__restrict__ fbx, const double *__restrict__ fby, long nx,
                      int ny, const uint8_t *__restrict__ mask, double dt, double hx,
                      double hy, int sources, int time_dg, const DevPar &Pv, const Consts &C,
                      const Batch &B, int parts, long c, int g, bool inrange, long fbase) {
  constexpr int V = L::V;
  constexpr int NS = ND == 1 ? NN : NN * NN;
  constexpr int NP = NN * NS;
  constexpr int XB = ND == 1 ? 1 : 2;
  constexpr int YB = 1;
  long ncell = ND == 1 ? nx : (long)nx * ny;
  bool valid = inrange && c < ncell;
  long cc = valid ? c : 0;
  const int inst = BATCH ? B.inst_u[cc] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  long ci = ND == 1 ? cc : (cc / ny);
  int cj = ND == 1 ? 0 : (int)(cc % ny);
  long cb = ND == 1 ? ci + 1 : (long)(ci + 1) * (ny + 2) + (cj + 1);
  long fo = ci;  // face on the left of the cell (1D)
  if (BATCH) {
    long li = cc - B.off_u[inst];
    cb = B.off_b[inst] + li + 1;
    fo = B.off_f[inst] + li;
    dt = B.clk[5 * inst + 1];
    hx = B.idx[inst] * C.derv[0][1];
  }
  bool active = valid && (mask == nullptr || mask[cb]);
  // a warp of masked-off cells writes nothing (800 x 400, two materials: the
  // two cell passes go from 1.58 to 0.82 ms)
  if (!__any_sync(0xffffffffu, active))
    return;
  int t = g / NS, sidx = g % NS;
  int i = ND == 1 ? sidx : sidx / NN, j = ND == 1 ? 0 : sidx % NN;
  int nt = time_dg ? NN : 1;
  bool live = active && (time_dg || t == 0);
  int tt = time_dg ? t : 0;
  const double *qc = qh + ((cb * nt + tt) * NS + sidx) * V;
  double q[V], acc[V];
#pragma unroll
  for (int k = 0; k < V; k++)
    acc[k] = 0.0;
  if (parts & FV_CENTERS) {
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = qc[k];
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(q, P, s);
    // wn (S - B dq/dx [- B dq/dy]), wn folded into the source's scalar
    // factors and the derivative coefficients (B is linear)
    const double wn = dt * ((time_dg ? GAUSS_W : 1.0) * (ND == 1 ? GAUSS_W : GAUSS_W * GAUSS_W));
    if (sources)
      source<L::THERMAL, V>(q, s, P, acc, wn);
    // - B dq by the node lines' differences, as dg_residual
#pragma unroll
    for (int d = 0; d < ND; d++) {
      const int lm = d == 0 ? XB : YB;
      const double h = d == 0 ? hx : hy;
      const double cf = wn * ((d == 0 ? i : j) ? -h : h);
      const double vc[3] = {s.v[0] * cf, s.v[1] * cf, s.v[2] * cf};
#pragma unroll
      for (int k = 5; k < V; k++) {
        const bool lset = k >= V - L::LSET;
        if (!lset && (k >= 14 || (k - 5) % 3 == d))
          continue;
        const double df = __shfl_xor_sync(0xffffffffu, q[k], lm) - q[k];
        acc[k] = fma(-vc[d], df, acc[k]);
        if (!lset) {
          const int col = (k - 5) % 3, dst = k - col + d;
          acc[dst] = fma(vc[col], df, acc[dst]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < V; k++)
      acc[k] = live ? acc[k] : 0.0;
  }
  // the cell's sum over its NP lanes, scattered: lane g holds variables
  // g CK .. g CK + CK - 1
  constexpr int CK = (V + NP - 1) / NP;
  double red[CK * NP];
#pragma unroll
  for (int k = 0; k < CK * NP; k++)
    red[k] = k < V ? acc[k] : 0.0;
  if (parts & FV_CENTERS)
    GroupReduceScatter<CK * NP, NP>::run(red, g);
  else {
#pragma unroll
    for (int k = 0; k < CK; k++)
      red[k] = 0.0;
  }
  if (!valid || !active)
    return;
  const bool faces = parts & FV_INTERFS;
  double *uc = u + cc * V;
  if (ND == 1) {
    // face ci: R part, face ci+1: L part (fv.cpp:143-146)
    const double *fl = fbx + (fo - fbase) * 2 * V;
    const double *fr = fbx + (fo - fbase + 1) * 2 * V;
    bool okl = mask == nullptr || (mask[cb - 1] && mask[cb]);
    bool okr = mask == nullptr || (mask[cb] && mask[cb + 1]);
#pragma unroll
    for (int p = 0; p < CK; p++) {
      const int k = g * CK + p;
      if (k >= V)
        break;
      double x = uc[k] + red[p];
      if (faces && okr)
        x -= fr[k];
      if (faces && okl)
        x -= fl[V + k];
      uc[k] = x;
    }
  } else {
    // x faces (fi, fj) with fi = ci+1 (L part) and fi = ci (R part), fj = cj+1;
    // y faces fi = ci+1 with fj = cj+1 (L part) and fj = cj (R part).
    long fxl = (long)(ci + 1) * (ny + 1) + (cj + 1);  // L part to this cell
    long fxr = (long)ci * (ny + 1) + (cj + 1);        // R part to this cell
    long fyl = (long)(ci + 1) * (ny + 1) + (cj + 1);
    long fyr = (long)(ci + 1) * (ny + 1) + cj;
#pragma unroll
    for (int p = 0; p < CK; p++) {
      const int k = g * CK + p;
      if (k >= V)
        break;
      double x = uc[k] + red[p];
      if (faces) {
        x -= fbx[fxl * 2 * V + k];
        x -= fbx[fxr * 2 * V + V + k];
        x -= fby[fyl * 2 * V + k];
        x -= fby[fyr * 2 * V + V + k];
      }
      uc[k] = x;
    }
  }
}

template <class L, int ND, bool BATCH = false>
__global__ void __launch_bounds__(128) k_cells(
    double *__restrict__ u, const double *__restrict__ qh, const double *__restrict__ fbx,
    const double *__restrict__ fby, long nx, int ny, const uint8_t *__restrict__ mask,
    double dt, const double *__restrict__ dt_dev, double hx, double hy, int sources,
    int time_dg, DevPar Pv, Consts C, Batch B, int parts) {
  constexpr int NP = NN * (ND == 1 ? NN : NN * NN);
  if (dt_dev)
    dt = *dt_dev;
  long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  cells_body<L, ND, BATCH>(u, qh, fbx, fby, nx, ny, mask, dt, hx, hy, sources, time_dg, Pv, C,
                           B, parts, gt / NP, threadIdx.x % NP, true, 0);
}

// The whole 1D FV update of fv_launcher (centers1 + interfs1, fv.cpp:11-160)
// in one launch, Rusanov flux: a block takes a tile of TILE cells; its
// 4 (TILE + 1) threads first evaluate the tile's TILE + 1 faces (one lane per
// face, time node and side, as k_faces1d_split) into shared memory, then
// the cells' volume terms (one lane per space-time node, as k_cells), and
// each cell's lanes apply u += volume - its two faces' contributions.  A
// face between two tiles is evaluated by both (one face in TILE + 1 twice);
// the sums and their order are those of the two-launch form.
// A small grid takes tiles of FV1_TILE_SMALL cells (one warp per block), so
// that its few warps run on separate SMs.
constexpr int FV1_TILE = 31;
constexpr int FV1_TILE_SMALL = 7;
template <class L, int TILE = FV1_TILE>
__global__ void __launch_bounds__(128) k_fv1d(
    double *__restrict__ u, const double *__restrict__ qh, long nx,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double idx,
    int sources, int time_dg, DevPar P, Consts C, int parts) {
  constexpr int V = L::V;
  static_assert(NN == 2 && 4 * (TILE + 1) <= 128 && (TILE + 1) % 8 == 0,
                "four lanes per face and per cell, whole warps");
  __shared__ double sfb[(TILE + 1) * 2 * V];
  if (dt_dev)
    dt = *dt_dev;
  const long c0 = (long)blockIdx.x * TILE;  // first cell, and first face, of the tile
  const int slot = threadIdx.x >> 2, lq = threadIdx.x & 3;
  if (parts & FV_INTERFS)
    faces1d_split_body<L, false>(sfb, qh, nx + 1, mask, dt, idx, time_dg, P, C, Batch{},
                                 c0 + slot, lq, true, c0);
  __syncthreads();
  cells_body<L, 1, false>(u, qh, sfb, nullptr, nx, 1, mask, dt, idx * C.derv[0][1], 0.0,
                          sources, time_dg, P, C, Batch{}, parts, c0 + slot, lq, slot < TILE, c0);
}

// ---------------------------------------------------------------------------
// Device clock of the device-resident time loop: [t, dt, tf, cfl, count].
// clock_dt reads t/count and writes dt from the CFL maximum (0 once t >= tf);
// clock_step adds dt to t and counts the step.
GPR_D void clock_dt(unsigned long long mx, double *__restrict__ clk) {
  double t = clk[0], tf = clk[2], cfl = clk[3];
  long count = (long)clk[4];
  double dt = 0.0;
  if (t < tf) {
    double MAX = __longlong_as_double((long long)mx);
    dt = cfl / MAX;
    if (count <= 5)
      dt *= 0.2;
    if (t + dt > tf)
      dt = tf - t;
  }
  clk[1] = dt;
}
GPR_D void clock_step(double *__restrict__ clk) {
  if (clk[1] > 0.0) {
    clk[0] += clk[1];
    clk[4] += 1.0;
  }
}
static __global__ void k_clock_finalize(const unsigned long long *__restrict__ mx,
                                        double *__restrict__ clk) {
  clock_dt(*mx, clk);
}
static __global__ void k_clock_advance(double *__restrict__ clk) { clock_step(clk); }

// CFL time step (solvers/iterator.cpp:54-83): per-cell sum_d mae/dx_d,
// block max, atomicMax on the bit pattern (non-negative doubles order as
// unsigned integers); NaN cells are skipped as std::max skips them.
// With clk the last block to finish (out[1]: the step's contortion flag, cleared
// here, and the blocks' counter) sets the clock's dt, which saves a launch of
// one thread (3.6 us in the 200-cell tube's step of 180).
template <class L>
__global__ void __launch_bounds__(256) k_cfl_max(const double *__restrict__ u, long ncell,
                                                 int nd, double idx, double idy,
                                                 unsigned long long *__restrict__ out,
                                                 DevPar P, double *__restrict__ clk = nullptr) {
  constexpr int V = L::V;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  double m = 0.0;
  if (c < ncell) {
    double q[V];
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = u[c * V + k];
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(q, P, s);
    double tmp = max_abs_eigs<L::THERMAL>(q, s, 0, P) * idx;
    if (nd == 2)
      tmp = fma(max_abs_eigs<L::THERMAL>(q, s, 1, P), idy, tmp);
    if (tmp > m)
      m = tmp;
  }
#pragma unroll
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
    if (clk) {
      int *flag = (int *)(out + 1), *count = flag + 1;
      __threadfence();
      if (atomicAdd(count, 1) == (int)gridDim.x - 1) {
        __threadfence();
        *flag = *count = 0;
        clock_dt(atomicMax(out, 0ull), clk);
      }
    }
  }
}

static __global__ void k_cfl_finalize(const unsigned long long *__restrict__ mx, double cfl, double t,
                               double tf, int count, double *__restrict__ dt_out) {
  double MAX = __longlong_as_double((long long)*mx);
  double dt = cfl / MAX;
  if (count <= 5)
    dt *= 0.2;
  if (t + dt > tf)
    dt = tf - t;
  *dt_out = dt;
}

// *flag = 1 if any of the n entries is a NaN (integer tests on the bit patterns).
static __global__ void k_any_nan(const double *__restrict__ u, long n, double *__restrict__ flag) {
  bool found = false;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
       i += (long)gridDim.x * blockDim.x)
    found = found || fp_abs_bits(u[i]) > FP_INF_BITS;
  if (found)
    *flag = 1.0;
}

// renorm_distortion (solvers/utils.cpp:6-23); skipped when the device clock
// says the step did not run (dt == 0).
template <int V>
__global__ void k_renorm(double *__restrict__ u, long ncell, double rho0,
                         const double *__restrict__ dt_dev) {
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  if (dt_dev && *dt_dev == 0.0)
    return;
  double *q = u + c * V;
  double r = q[0];
  if (r > 0) {
    double A[9];
#pragma unroll
    for (int k = 0; k < 9; k++)
      A[k] = q[5 + k];
    double f = cbrt(r / (rho0 * det3(A)));
#pragma unroll
    for (int k = 0; k < 9; k++)
      q[5 + k] = A[k] * f;
  }
}

// k_renorm followed by the contortion test of the renormalised cell
// (contorted, solvers/utils.cpp:66-85, as k_contorted): one launch for both.
template <int V>
__global__ void k_renorm_contorted(double *__restrict__ u, long ncell, double rho0, double tol,
                                   int *__restrict__ flag, const double *__restrict__ dt_dev) {
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  if (dt_dev && *dt_dev == 0.0)
    return;
  double *q = u + c * V;
  double A[9];
#pragma unroll
  for (int k = 0; k < 9; k++)
    A[k] = q[5 + k];
  const double r = q[0];
  if (r > 0) {
    double f = cbrt(r / (rho0 * det3(A)));
#pragma unroll
    for (int k = 0; k < 9; k++) {
      A[k] *= f;
      q[5 + k] = A[k];
    }
  }
  double f2 = 0.0;
#pragma unroll
  for (int k = 0; k < 9; k++)
    f2 += A[k] * A[k];
  double d13 = cbrt(fabs(det3(A)));
  if (f2 / (3.0 * d13 * d13) - 1.0 > tol)
    atomicOr(flag, 1);
}

// ---------------------------------------------------------------------------
// Batched helper kernels (1D).

// ub of every instance: interior copy and ghost cells (grid.cpp:12-125,
// 147-160), one thread per (packed ub cell, variable).
template <int V>
__global__ void k_b_boundaries(const double *__restrict__ u, double *__restrict__ ub,
                               long nub, Batch B) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= nub * V)
    return;
  int k = idx % V;
  long cb = idx / V;
  int inst = B.inst_ub[cb];
  int nx = B.nx[inst];
  long li = cb - B.off_ub[inst];
  const double *ui = u + (long)B.off_u[inst] * V;
  if (li >= NN && li < nx + NN) {
    ub[cb * V + k] = ui[(li - NN) * V + k];
    return;
  }
  int side = li >= nx + NN;
  int gi = side ? (int)(li - nx - NN) : (int)li;
  int code = B.bc[2 * inst + side];
  int si = bc_src_index(code, side, gi, nx);
  if (code == GPR_BC_PERIODIC)
    code = GPR_BC_TRANSMISSIVE;
  ub[cb * V + k] = bc_value<V>(code, 0, k, ui + (long)si * V);
}

// WENO per (packed predictor cell, variable)
template <int V>
__global__ void k_b_weno(double *__restrict__ wh, const double *__restrict__ ub, long ncb,
                         Batch B) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (idx >= ncb * V)
    return;
  int k = idx % V;
  long c = idx / V;
  int inst = B.inst_b[c];
  long li = c - B.off_b[inst];
  const double *d0 = ub + ((long)B.off_ub[inst] + li) * V + k;
  weno_point(d0, V, wh + c * NN * V + k, V, (int)li, B.nx[inst] + 2, 0);
}

// per-instance CFL maximum: atomicMax of the bit pattern per instance
template <class L>
__global__ void __launch_bounds__(256) k_b_cfl_max(const double *__restrict__ u, long ncell,
                                                   unsigned long long *__restrict__ mx,
                                                   Batch B, double *__restrict__ mcell = nullptr) {
  constexpr int V = L::V;
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  int inst = B.inst_u[c];
  const DevPar &P = B.P[inst];
  double q[V];
#pragma unroll
  for (int k = 0; k < V; k++)
    q[k] = u[c * V + k];
  Prim<L::THERMAL> s;
  prim<L::THERMAL>(q, P, s);
  double m = max_abs_eigs<L::THERMAL>(q, s, 0, P) * B.idx[inst];
  if (mcell)
    mcell[c] = m;
  if (m > 0.0)  // NaN and zero are skipped
    atomicMax(mx + inst, (unsigned long long)__double_as_longlong(m));
}

// per-instance dt (iterator.cpp:54-83 per instance) and the step counter
static __global__ void k_b_clock_finalize(unsigned long long *__restrict__ mx, Batch B) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= B.ninst)
    return;
  double *c = B.clk + 5 * k;
  double t = c[0], tf = c[2], cfl = c[3];
  long count = (long)c[4];
  double dt = 0.0;
  if (t < tf) {
    double MAX = __longlong_as_double((long long)mx[k]);
    dt = cfl / MAX;
    if (count <= 5)
      dt *= 0.2;
    if (t + dt > tf)
      dt = tf - t;
  }
  c[1] = dt;
  mx[k] = 0ull;  // ready for the next step's maximum
}

template <int V>
__global__ void k_b_renorm(double *__restrict__ u, long ncell, Batch B) {
  long c = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (c >= ncell)
    return;
  int inst = B.inst_u[c];
  if (B.clk[5 * inst + 1] == 0.0)
    return;
  double *q = u + c * V;
  double r = q[0];
  if (r > 0) {
    double A[9];
#pragma unroll
    for (int k = 0; k < 9; k++)
      A[k] = q[5 + k];
    double f = cbrt(r / (B.P[inst].rho0 * det3(A)));
#pragma unroll
    for (int k = 0; k < 9; k++)
      q[5 + k] = A[k] * f;
  }
}

static __global__ void k_b_clock_advance(Batch B, unsigned long long *__restrict__ updates) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= B.ninst)
    return;
  double *c = B.clk + 5 * k;
  if (c[1] > 0.0) {
    c[0] += c[1];
    c[4] += 1.0;
    if (updates)
      atomicAdd(updates, (unsigned long long)B.nx[k]);
  }
}

}  // namespace gpr
