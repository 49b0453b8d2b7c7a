// Design-side kernels of one OC iteration: the hat-weight filters, the
// compliance/sensitivity kernel and the device-side OC bisection.
#pragma once

#include <cmath>

#include "common.cuh"

namespace tpo {

// ---------------------------------------------------------------------------
// Hat-weight filter (reference optimizer/filter.py:22-171).
// The reference precomputes a neighbour list on the host; here each CTA
// derives the weights w(dx,dy) = rmin - sqrt(dx^2+dy^2) for the
// (2R+1)^2 box (R = ceil(rmin)) into shared memory, stages a 32x32 element
// tile plus an R-wide halo, and sums in the reference's neighbour order
// (dx outer, dy inner), skipping w <= 0 and out-of-domain neighbours.
// ---------------------------------------------------------------------------
constexpr int FT = 32;           // tile edge (elements)
constexpr int F_THREADS = 128;   // radii up to F_REGR
constexpr int FA_THREADS = 256;  // larger radii
constexpr int F_REGR = 8;
constexpr int F_MAXR = 16;

enum FilterMode { F_DENSITY = 0, F_SENS = 1 };

// largest |dy| with a positive weight beside |dx| (-1: none)
__device__ __forceinline__ int filter_chord(double rmin, int dx, int R) {
  int m = -1;
  for (int dy = 0; dy <= R; ++dy)
    if (rmin - sqrt((double)(dx * dx + dy * dy)) > 0.0) m = dy;
  return m;
}

// Radii from F_REGR + 1 to F_MAXR. (bx, by) = (tile row, tile column) of this CTA.
// Bound by two shared loads per neighbour and by the warps that cover their latency:
// a tile of 21 to 41 KB limits the CTAs of an SM, so a CTA has 256 threads, in a
// kernel without the register form's 78 registers. A row of the box is its chord of
// positive weights inside the grid, without a test per neighbour. Density filter of
// 517x173 elements at R = 9, 12, 16: 36, 51, 78 us (47, 67, 105 with the tests; 80,
// 114, 179 with 128 threads and both forms in one kernel).
template <int MODE>
__device__ __forceinline__ void filter_any(int nx, int ny, double rmin, int R,
                                           const double *__restrict__ x,
                                           const double *__restrict__ rho,
                                           double *__restrict__ out, double *__restrict__ s_out,
                                           float *__restrict__ s32_out, double e_min, double pen,
                                           int bx, int by) {
  extern __shared__ double fsm[];
  const int W = 2 * R + 1;
  const int TW = FT + 2 * R;  // staged tile edge
  double *wt = fsm;           // W*W weights
  double *tile = fsm + W * W; // TW*TW values, index tx*TW + ty
  __shared__ int chord[F_MAXR + 1];  // largest |dy| with a positive weight (-1: none)
  const int ex0 = by * FT, ey0 = bx * FT;

  if (threadIdx.x <= R) chord[threadIdx.x] = filter_chord(rmin, threadIdx.x, R);
  for (int k = threadIdx.x; k < W * W; k += blockDim.x) {
    const int dx = k / W - R, dy = k % W - R;
    wt[k] = rmin - sqrt((double)(dx * dx + dy * dy));
  }
  for (int k = threadIdx.x; k < TW * TW; k += blockDim.x) {
    const int tx = k / TW, ty = k % TW;
    const int gx = ex0 - R + tx, gy = ey0 - R + ty;
    double v = 0.0;
    if (gx >= 0 && gx < nx && gy >= 0 && gy < ny) {
      const size_t e = (size_t)gx * ny + gy;
      v = (MODE == F_SENS) ? rho[e] * x[e] : x[e];
    }
    tile[k] = v;
  }
  __syncthreads();

  const int ty = threadIdx.x & 31;
  const int ey = ey0 + ty;
  for (int tx = threadIdx.x >> 5; tx < FT; tx += FA_THREADS / 32) {
    const int ex = ex0 + tx;
    if (ex >= nx || ey >= ny) continue;
    double num = 0.0, den = 0.0;
    for (int dx = -R; dx <= R; ++dx) {
      const int jx = ex + dx;
      if (jx < 0 || jx >= nx) continue;
      const double *trow = tile + (size_t)(tx + R + dx) * TW + (ty + R);
      const double *wrow = wt + (dx + R) * W + R;
      const int m = chord[abs(dx)], d1 = min(m, ny - 1 - ey);
#pragma unroll 4
      for (int dy = max(-m, -ey); dy <= d1; ++dy) {
        const double w = wrow[dy];
        num = fma(w, trow[dy], num);
        den += w;
      }
    }
    const size_t e = (size_t)ex * ny + ey;
    double o;
    if (MODE == F_SENS) {
      o = num / (rho[e] * den + 1e-20);
    } else {
      o = num / (den + 1e-20);
      if (s_out || s32_out) {
        const double s = e_min + pow(o, pen) * (1.0 - e_min);
        if (s_out) s_out[e] = s;
        if (s32_out) s32_out[e] = (float)s;
      }
    }
    out[e] = o;
  }
}
// Radii up to F_REGR: F_ROWS rows of a column per thread. For every column dx
// of the box a thread reads the 2 R + F_ROWS values its rows need once (16-byte
// shared loads, conflict-free by the pitch) and the R + 1 weights, and adds the
// chord of positive weights, instead of two shared loads and two tests per
// neighbour: at rmin = 4 about 10 loads per element instead of 162. An element
// whose box lies inside the grid takes the weight sum den_in (filter_den).
// Values and weights are added in the reference's order (dx, then dy). At rmin = 4
// on 2048x1024 elements 96 -> 33 us (46 us with the tile staged one load at a time).
// F_SENS keeps the tile's own rho from the staging: its last division read it again
// lane by column, a third of the time at R = 1 (29.1 -> 20.7 us; R = 4 39.7 -> 32.9).
constexpr int F_ROWS = 8;
static_assert(F_THREADS / 32 * F_ROWS == FT, "a CTA covers the tile");
template <int MODE, int R>
__device__ __forceinline__ void filter_reg(int nx, int ny, double rmin,
                                           const double *__restrict__ x,
                                           const double *__restrict__ rho,
                                           double *__restrict__ out, double *__restrict__ s_out,
                                           float *__restrict__ s32_out, double e_min, double pen,
                                           double den_in, int bx, int by) {
  constexpr int RA = (R + 1) / 2 * 2, TH = FT + 2 * RA, PITCH = TH + 2, TC = FT + 2 * R;
  constexpr int NV = 2 * RA + F_ROWS;
  static_assert(PITCH % 4 == 2, "16-byte loads of eight lanes fall into distinct banks");
  extern __shared__ __align__(16) double fsm[];
  double *tile = fsm;               // [TC][PITCH], rows from ey0 - RA
  double *wt = fsm + TC * PITCH;    // [R + 1][R + 1] by |dx|, |dy|
  double *own = wt + (R + 1) * (R + 1);  // F_SENS: rho of the tile itself, [FT][FT + 1]
  __shared__ int chord[R + 1];      // largest |dy| with a positive weight (-1: none)
  const int ex0 = by * FT, ey0 = bx * FT;
  for (int k = threadIdx.x; k < (R + 1) * (R + 1); k += F_THREADS) {
    const int dx = k / (R + 1), dy = k % (R + 1);
    wt[k] = rmin - sqrt((double)(dx * dx + dy * dy));
  }
  if (threadIdx.x <= R) chord[threadIdx.x] = filter_chord(rmin, threadIdx.x, R);
  constexpr int NB = 8;  // loads in flight per thread
  for (int k0 = threadIdx.x; k0 < TC * TH; k0 += NB * F_THREADS) {
    double v[NB], q[MODE == F_SENS ? NB : 1];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int k = k0 + i * F_THREADS, tx = k / TH, ty = k - tx * TH;
      const int gx = ex0 - R + tx, gy = ey0 - RA + ty;
      v[i] = 0.0;
      if (MODE == F_SENS) q[i] = 0.0;
      if (k < TC * TH && gx >= 0 && gx < nx && gy >= 0 && gy < ny) {
        const size_t e = (size_t)gx * ny + gy;
        v[i] = x[e];
        if (MODE == F_SENS) q[i] = rho[e];
      }
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int k = k0 + i * F_THREADS, tx = k / TH, ty = k - tx * TH;
      if (k < TC * TH) {
        tile[tx * PITCH + ty] = MODE == F_SENS ? q[i] * v[i] : v[i];
        if (MODE == F_SENS && (unsigned)(tx - R) < FT && (unsigned)(ty - RA) < FT)
          own[(tx - R) * (FT + 1) + ty - RA] = q[i];
      }
    }
  }
  __syncthreads();

  const int tx = threadIdx.x & 31, r0 = F_ROWS * (threadIdx.x >> 5);
  const int ex = ex0 + tx, ey = ey0 + r0;
  if (ex >= nx || ey >= ny) return;
  double num[F_ROWS], den[F_ROWS];
#pragma unroll
  for (int j = 0; j < F_ROWS; ++j) {
    num[j] = 0.0;
    den[j] = den_in;
  }
#pragma unroll 1
  for (int dx = -R; dx <= R; ++dx) {
    const int m = chord[abs(dx)];
    if (m < 0) continue;
    const double2 *col = reinterpret_cast<const double2 *>(tile + (tx + R + dx) * PITCH + r0);
    const double *w = wt + abs(dx) * (R + 1);
    double v[NV];
#pragma unroll
    for (int i = 0; i < NV / 2; ++i) {
      const double2 q = col[i];
      v[2 * i] = q.x;
      v[2 * i + 1] = q.y;
    }
#pragma unroll
    for (int d = -R; d <= R; ++d) {
      if (abs(d) <= m) {
        const double wd = w[abs(d)];
#pragma unroll
        for (int j = 0; j < F_ROWS; ++j) num[j] = fma(wd, v[RA + j + d], num[j]);
      }
    }
  }
  const bool inner = ex >= R && ex + R < nx && ey >= R && ey + F_ROWS - 1 + R < ny;
  if (!inner) {  // the weights inside the grid, in the same order
#pragma unroll
    for (int j = 0; j < F_ROWS; ++j) den[j] = 0.0;
    for (int dx = max(-R, -ex); dx <= min(R, nx - 1 - ex); ++dx) {
      const int m = chord[abs(dx)];
      for (int dy = -m; dy <= m; ++dy) {
        const double wd = wt[abs(dx) * (R + 1) + abs(dy)];
#pragma unroll
        for (int j = 0; j < F_ROWS; ++j)
          den[j] += (unsigned)(ey + j + dy) < (unsigned)ny ? wd : 0.0;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < F_ROWS; ++j) {
    const int yj = ey + j;
    if (yj >= ny) break;
    const size_t e = (size_t)ex * ny + yj;
    double o;
    if (MODE == F_SENS) {
      o = num[j] / (own[tx * (FT + 1) + r0 + j] * den[j] + 1e-20);
    } else {
      o = num[j] / (den[j] + 1e-20);
      if (s_out || s32_out) {
        const double s = e_min + pow(o, pen) * (1.0 - e_min);
        if (s_out) s_out[e] = s;
        if (s32_out) s32_out[e] = (float)s;
      }
    }
    out[e] = o;
  }
}

// sum of the positive weights of a whole box, in the order dx, dy
inline double filter_den(double rmin, int R) {
  double d = 0.0;
  for (int dx = -R; dx <= R; ++dx)
    for (int dy = -R; dy <= R; ++dy) {
      const double w = rmin - std::sqrt((double)(dx * dx + dy * dy));
      if (w > 0.0) d += w;
    }
  return d;
}

// dynamic shared memory of a filter launch
inline int filter_smem_bytes(int R, int mode = F_DENSITY) {
  const int W = 2 * R + 1, TW = FT + 2 * R, RA = (R + 1) / 2 * 2;
  if (R > F_REGR) return (W * W + TW * TW) * (int)sizeof(double);
  const int own = mode == F_SENS ? FT * (FT + 1) : 0;
  return (TW * (FT + 2 * RA + 2) + (R + 1) * (R + 1) + own) * (int)sizeof(double);
}

template <int MODE>
__device__ __forceinline__ void filter_run(int nx, int ny, double rmin, int R,
                                           const double *__restrict__ x,
                                           const double *__restrict__ rho,
                                           double *__restrict__ out, double *__restrict__ s_out,
                                           float *__restrict__ s32_out, double e_min, double pen,
                                           double den, int bx, int by) {
  switch (R) {
#define TPO_F(r)                                                                          \
  case r:                                                                                 \
    filter_reg<MODE, r>(nx, ny, rmin, x, rho, out, s_out, s32_out, e_min, pen, den, bx,   \
                        by);                                                              \
    break;
    TPO_F(1) TPO_F(2) TPO_F(3) TPO_F(4) TPO_F(5) TPO_F(6) TPO_F(7) TPO_F(8)
#undef TPO_F
  }
}
template <int MODE>
__global__ void __launch_bounds__(F_THREADS)
    k_filter(int nx, int ny, double rmin, int R, const double *__restrict__ x,
             const double *__restrict__ rho, double *__restrict__ out,
             double *__restrict__ s_out, float *__restrict__ s32_out, double e_min, double pen,
             double den) {
  filter_run<MODE>(nx, ny, rmin, R, x, rho, out, s_out, s32_out, e_min, pen, den, blockIdx.x,
                   blockIdx.y);
}
template <int MODE>
__global__ void __launch_bounds__(FA_THREADS)
    k_filter_any(int nx, int ny, double rmin, int R, const double *__restrict__ x,
                 const double *__restrict__ rho, double *__restrict__ out,
                 double *__restrict__ s_out, float *__restrict__ s32_out, double e_min,
                 double pen) {
  filter_any<MODE>(nx, ny, rmin, R, x, rho, out, s_out, s32_out, e_min, pen, blockIdx.x,
                   blockIdx.y);
}

// ---------------------------------------------------------------------------
// Compliance and sensitivity (reference fem/kernels.py:234-272):
//   uKu_e = u_e^T Ke u_e, dc_e = -p rho_e^(p-1) (1 - e_min) uKu_e,
//   c = sum_e (e_min + rho_e^p (1 - e_min)) uKu_e.
// One element per thread and step, a few elements in flight per thread's loop:
// a thread that walked 16 columns with two pow per element took 33 us even on
// 1200 elements (80 us at 2048x1024). The dense product keeps the
// order of its sums: uKu cancels from |u|^2 down to the squared strains, so
// another order moves dc by 1e-11 on a 2048-element span.
// The product is a function call: inlined, the loop keeps Ke's 64 entries in 128
// registers (or, held at 64, spills them: 276 bytes a thread), where the function
// takes them as constant operands and leaves 48. Inlined and spilled / inlined at
// 128 registers / called: 69.9, 51.9, 40.0 us at 2048x1024, 24.4, 18.6, 14.4 at
// 3x100000 (the column march of before: 65.7, 20.6).
// ---------------------------------------------------------------------------
constexpr int S_THREADS = 256;

__device__ __noinline__ double elem_energy(double2 bl, double2 br, double2 tr, double2 tl) {
  const double ue[8] = {bl.x, bl.y, br.x, br.y, tr.x, tr.y, tl.x, tl.y};
  double uku = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    double ku = c_ke[i * 8] * ue[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) ku = fma(c_ke[i * 8 + j], ue[j], ku);
    uku = fma(ue[i], ku, uku);
  }
  return uku;
}

__device__ __forceinline__ void sensitivity_run(int nx, int ny, double e_min, double pen,
                                                const double *__restrict__ rho,
                                                const double *__restrict__ u,
                                                double *__restrict__ dc, double *part, SumCtl *ctl,
                                                double *c_out, int nb, int bid) {
  const int n = nx * ny;
  const double2 *__restrict__ un = reinterpret_cast<const double2 *>(u);
  double acc[1] = {0.0};
  for (int e = bid * S_THREADS + threadIdx.x; e < n; e += nb * S_THREADS) {
    const int ex = e / ny;
    const double2 *q = un + (e + ex);  // node (ex, ey) of ny + 1 rows
    const double uku = elem_energy(q[0], q[ny + 1], q[ny + 2], q[1]);
    const double r = rho[e];
    dc[e] = -pen * pow(r, pen - 1.0) * (1.0 - e_min) * uku;
    acc[0] += (e_min + simp_pow(r, pen) * (1.0 - e_min)) * uku;
  }
  if (!grid_reduce<1>(acc, part, &ctl->counter, nb, bid)) return;
  if (threadIdx.x == 0) *c_out = acc[0];
}
__global__ void __launch_bounds__(S_THREADS, 5)
    k_sensitivity(int nx, int ny, double e_min, double pen, const double *__restrict__ rho,
                  const double *__restrict__ u, double *__restrict__ dc, double *part,
                  SumCtl *ctl, double *c_out) {
  sensitivity_run(nx, ny, e_min, pen, rho, u, dc, part, ctl, c_out, gridDim.x, blockIdx.x);
}

// ---------------------------------------------------------------------------
// OC update (reference optimizer/oc.py:21-93): bisection on lambda in [0, 1e9],
// at most OC_MAX_STEPS midpoints, stop when (hi - lo)/(hi + lo + 1e-30) < 1e-4;
// the density of the last midpoint evaluated. One launch: the CTAs stay
// resident and lambda never visits the host.
//
// One midpoint per pass over the elements (a launch each, with a division and
// a square root per element) took 978 us for the 2048x1024 bridge and 400 us
// for 517x173: 50 passes, bound by their latency and the FP64 division. An OC
// iteration without its solve went from 1098 to 346 us and from 457 to 91 us
// with this form. A pass evaluates OC_NL = 7 values of lambda:
// * While every midpoint so far has been an upper bound, the midpoints are
//   1e9 / 2^k whatever the data. The volume falls as lambda grows, so the
//   first k whose volume exceeds the target is found by two passes (every 7th
//   k, then the six between).
// * After that (and always when dv is given, whose sign could make the volume
//   rise) a pass evaluates the three next levels of the bisection tree, the
//   seven midpoints the next three steps can visit, and walks it.
// The midpoints, their order, the stop test and the step count are those of
// the one-at-a-time bisection. At most 7 passes instead of 50; with dv, where every
// level is walked, at most 17 (25 on large designs, below).
// With dv = 1 the candidate is rho sqrt(-dc / (lambda + 1e-20)), so a pass needs
// s = rho sqrt(-dc) once and then a multiplication by 1 / sqrt(lambda + 1e-20),
// two comparisons and an addition per lambda. (1e-20 is not lost beside lambda:
// from 1e9 / 2^43 down, the 43rd midpoint, it is part of the sum.) s stays
// in registers (up to OC_EPT elements per thread) or in `sbuf` (n doubles).
// The density, its mean and the largest change come from the formula itself.
// With dv every value of lambda costs a division and a square root, and on large
// designs their number is the time, not the passes. Beyond OC_DV_EPT elements per
// thread a pass evaluates two levels of the tree: 75 values in 25 passes instead of
// 119 in 17. Two levels / three: 176, 154 us at 303,104 elements, 221, 226 at 500,000,
// 248, 257 at 700,000, 471, 577 at 2.1 M, 1.75, 2.12 ms at 8 M, 6.3, 8.0 ms at 32 M
// (7.7 there with a launch per midpoint).
// ---------------------------------------------------------------------------
constexpr int OC_THREADS = 1024;
constexpr int OC_MAX_STEPS = 50;
constexpr int OC_NL = 7;
constexpr int OC_EPT = 2;
constexpr int OC_DV_EPT = 4;

__device__ __forceinline__ double oc_candidate(double r, double d, double dvv, double lam,
                                               double move) {
  const double be = fmax(-d / (lam * dvv + 1e-20), 0.0);
  const double cand = r * sqrt(be);
  const double lo = fmax(0.001, r - move);
  const double hi = fmin(1.0, r + move);
  return fmax(lo, fmin(hi, cand));
}

// the seven values of lambda of a pass and what the walk over their volumes decides
struct OcWalk {
  double lo, hi, last;
  int steps, scan, k0;  // scan: 1, 2 = locating the first k; 0 = tree
  bool done;
  __device__ __forceinline__ void init(bool monotone) {
    lo = 0.0;
    hi = 1e9;
    last = 0.0;
    steps = 0;
    scan = monotone ? 1 : 0;
    k0 = 0;
    done = false;
  }
  __device__ __forceinline__ double lam(int j) const {
    if (scan == 1) return ldexp(1e9, -OC_NL * (j + 1));
    if (scan == 2) return ldexp(1e9, -(k0 + min(j + 1, OC_NL - 1)));
    const double m = 0.5 * (lo + hi);  // heap order: 0; 1, 2; 3 .. 6
    if (j == 0) return m;
    const double ml = 0.5 * (lo + m), mh = 0.5 * (m + hi);
    switch (j) {
      case 1: return ml;
      case 2: return mh;
      case 3: return 0.5 * (lo + ml);
      case 4: return 0.5 * (ml + m);
      case 5: return 0.5 * (m + mh);
      default: return 0.5 * (mh + hi);
    }
  }
  // above: bit j set if the volume at value j exceeds the target; levels: of the tree, evaluated
  __device__ __forceinline__ void walk(unsigned above, int levels) {
    if (scan == 1) {
      const int j = above ? __ffs(above) - 1 : OC_NL;
      k0 = OC_NL * j;
      if (k0 >= OC_MAX_STEPS - 1) {  // never: all 50 midpoints are upper bounds
        last = ldexp(1e9, -OC_MAX_STEPS);
        hi = last;
        steps = OC_MAX_STEPS;
        done = true;
      }
      scan = 2;
      return;
    }
    if (scan == 2) {
      above &= (1u << (OC_NL - 1)) - 1;
      const int j = above ? __ffs(above) - 1 : OC_NL - 1;
      steps = k0 + j + 1;
      last = lo = ldexp(1e9, -steps);
      hi = ldexp(1e9, -(steps - 1));
      done = steps >= OC_MAX_STEPS;
      scan = 0;
      return;
    }
    // three levels; the stop tests' divisions do not depend on each other
    double l[3], h[3], m[3], a = lo, b = hi;
    bool stop[3];
    int j = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      m[i] = 0.5 * (a + b);
      const bool up = (above >> j) & 1u;
      if (up) a = m[i]; else b = m[i];
      j = 2 * j + (up ? 2 : 1);
      l[i] = a;
      h[i] = b;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) stop[i] = (h[i] - l[i]) / (h[i] + l[i] + 1e-30) < 1e-4;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (i < levels && !done) {
        lo = l[i];
        hi = h[i];
        last = m[i];
        steps += 1;
        done = stop[i] || steps >= OC_MAX_STEPS;
      }
  }
};
static_assert(OC_NL == 7 && OC_NL * OC_NL == OC_MAX_STEPS - 1, "the scan covers k = 1 .. 49");

// What warp 0 decides between two passes, for the whole CTA.
struct OcShared {
  OcWalk w;
  double lam[OC_NL];  // with dv: lambda; else 1 / sqrt(lambda + 1e-20)
};

// The update of one design by a team of co-resident CTAs of OC_THREADS
// threads. rho_out may be rho_in. HELD: every thread's elements fit in its
// registers (n <= size * OC_THREADS * OC_EPT); otherwise sbuf holds s.
template <bool HELD, typename Team>
__device__ __forceinline__ void oc_run(Team &team, int n, double volfrac, double move,
                                       const double *rho_in, const double *__restrict__ dc,
                                       const double *__restrict__ dv, double *sbuf,
                                       double *rho_out, double *result, OcShared &sh) {
  const int stride = team.size() * OC_THREADS;
  const int levels = !HELD && dv && n > OC_DV_EPT * stride ? 2 : 3;
  const int e0 = team.rank() * OC_THREADS + threadIdx.x;
  double hr[HELD ? OC_EPT : 1], hs[HELD ? OC_EPT : 1];
  if (HELD) {
#pragma unroll
    for (int i = 0; i < OC_EPT; ++i) {
      const int e = e0 + i * stride;
      hr[i] = hs[i] = 0.0;
      if (e < n) {
        hr[i] = rho_in[e];
        hs[i] = hr[i] * sqrt(fmax(-dc[e], 0.0));
      }
    }
  } else if (!dv) {
    for (int e = e0; e < n; e += stride) sbuf[e] = rho_in[e] * sqrt(fmax(-dc[e], 0.0));
  }
  // warp 0 walks over the last pass's volumes (nullptr: the start) and sets
  // up the next one's multipliers, one per lane
  auto decide = [&](const double *sum) {
    if (threadIdx.x < 32) {
      OcWalk w = sh.w;
      const unsigned above =
          __ballot_sync(FULL, sum && threadIdx.x < OC_NL && sum[threadIdx.x] / n > volfrac);
      if (sum) w.walk(above, levels);
      else w.init(dv == nullptr);
      if (threadIdx.x == 0) sh.w = w;
      if (threadIdx.x < OC_NL) {
        const double l = w.lam(threadIdx.x);
        sh.lam[threadIdx.x] = dv ? l : rsqrt(l + 1e-20);
      }
    }
    __syncthreads();
  };
  decide(nullptr);
  while (!sh.w.done) {
    double acc[OC_NL];
#pragma unroll
    for (int j = 0; j < OC_NL; ++j) acc[j] = 0.0;
    const double *il = sh.lam;
    auto add = [&](double r, double s) {
      const double lo = fmax(0.001, r - move);
      const double hi = fmin(1.0, r + move);
#pragma unroll
      for (int j = 0; j < OC_NL; ++j) {
        double c = s * il[j];
        c = c <= hi ? c : hi;  // a NaN candidate counts as hi, as fmin(hi, NaN) does
        acc[j] += c < lo ? lo : c;
      }
    };
    if (dv) {
      for (int e = e0; e < n; e += stride) {
        const double r = rho_in[e], d = dc[e], v = dv[e];
#pragma unroll
        for (int j = 0; j < OC_NL; ++j)
          if (j < 3 || levels == 3) acc[j] += oc_candidate(r, d, v, il[j], move);
      }
    } else if (HELD) {
#pragma unroll
      for (int i = 0; i < OC_EPT; ++i)
        if (e0 + i * stride < n) add(hr[i], hs[i]);
    } else {
#pragma unroll 4
      for (int e = e0; e < n; e += stride) add(rho_in[e], sbuf[e]);
    }
    const double *sum = team.template reduce<OC_NL>(acc);
    if (!sum) {
      if (result && team.rank() == 0 && threadIdx.x < 4) result[threadIdx.x] = nan("");
      return;
    }
    decide(sum);
  }
  const double lam = sh.w.last;
  double fin[2] = {0.0, 0.0};  // sum of the new densities, largest change
  for (int e = e0; e < n; e += stride) {
    const double r = rho_in[e];
    const double nw = oc_candidate(r, dc[e], dv ? dv[e] : 1.0, lam, move);
    fin[0] += nw;
    fin[1] = fmax(fin[1], fabs(nw - r));
    rho_out[e] = nw;
  }
  const double *tot = team.template reduce<2, 2u>(fin);
  if (result && team.rank() == 0 && threadIdx.x == 0) {
    result[0] = tot ? tot[1] : nan("");
    result[1] = tot ? tot[0] / n : nan("");
    result[2] = lam;
    result[3] = (double)sh.w.steps;
  }
  team.leave();
}

// one cluster (small designs): its barrier costs less than the grid's
template <bool HELD>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(OC_THREADS, 1)
    k_oc_cluster(int n, double volfrac, double move, const double *rho_in, const double *dc,
                 const double *dv, double *sbuf, double *rho_out, double *result) {
  __shared__ typename ClusterTeam<OC_NL>::Shared ts;
  __shared__ OcShared sh;
  ClusterTeam<OC_NL> team(ts);
  oc_run<HELD>(team, n, volfrac, move, rho_in, dc, dv, sbuf, rho_out, result, sh);
}

// cooperative grid, at most one CTA per SM; *bar zeroed before the launch
template <bool HELD>
__global__ void __launch_bounds__(OC_THREADS, 1)
    k_oc_grid(int n, double volfrac, double move, const double *rho_in, const double *dc,
              const double *dv, double *sbuf, double *rho_out, double *result, GridBar *bar,
              double *part) {
  __shared__ typename GridTeam<OC_NL>::Shared ts;
  __shared__ OcShared sh;
  GridTeam<OC_NL> team(ts, bar, part);
  oc_run<HELD>(team, n, volfrac, move, rho_in, dc, dv, sbuf, rho_out, result, sh);
}

}  // namespace tpo
