// A whole plain-FP64 solve in one launch, for grids whose PCG state fits on the
// chip: two nodes per thread, at most one CTA per SM (2D, point preconditioners;
// 592 groups of 30 rows by 8 columns, 142,080 nodes where the grid fills them, 124,881
// at 460x270); one thread-block cluster where 16 CTAs hold the grid (32 groups, 7,680
// nodes at most), a cooperative launch otherwise.
//
// On such a grid the one-launch-per-iteration form (k_cgstep) spends 14-16 us
// an iteration on latency: launch, filling the TMA ring, eleven columns one
// after another, and two dependent levels of reduction, while the vectors
// would fit in registers. Here r, s, p, x, u and w stay in registers for the
// whole solve, and the CTAs exchange once per iteration:
//   s = w + beta s, r -= alpha s, u = M^-1 r   on own nodes and the halo ring
//   w = K u on own nodes
//   publish the edge nodes' w and the sums gamma, delta, ||r||^2; collect the
//   halo's w and all sums -> alpha, beta, the stop rules
// The halo's r and s are kept redundantly, so that w is all that crosses, at
// the same moment as the sums.
//
// Same bits as k_cgstep (without TURN, as at all sizes near this one's). A PCG run
// on a 1e9 contrast amplifies a change of one rounding, so the arithmetic and the
// order of every sum are k_cgstep's:
// * A block is the work of one of its CTAs: a strip of L columns x 120 rows, in
//   up to four groups of 30 rows (one of its warps each). A group has a warp
//   here for every two columns of the strip and its two neighbours, lanes 0 and
//   31 the halo rows. A thread forms the elements right of its nodes
//   (elem_forces); the node sums add the same four corner forces in the same
//   order.
// * The sums run over the strip's columns in order for each row, then over the
//   rows by the same butterfly, then over the groups of a block, and the
//   blocks' sums the way its last CTA adds them.
//
// Exchange in a cluster: edge values and sums wait in each CTA's shared memory,
// one cluster barrier, and the readers fetch them from their owners.
// Exchange in a cooperative grid, without barriers: a double travels as one
// 16-byte store of {low word, epoch, high word, epoch}; the reader polls its
// word until both epochs are the current exchange's (the store's and the load's
// two elements are 8-byte accesses, each single-copy atomic, so data and epoch
// arrive together). One store and one
// load latency instead of fence + arrive + poll + read. Two buffers by parity
// of the epoch suffice: a CTA publishes exchange e + 2 only after it has all
// sums of e + 1, which each CTA publishes after it has read all it needs of e.
// The words are zeroed before the launch; epochs start at 1. Sums are written
// to 16 copies, each polled by a sixteenth of the CTAs: with one copy all CTAs
// poll the same few cache lines, and the stores they wait for queue behind the
// polls (0.8 us an iteration at 400x200). With more than RES_ALL_UNITS units
// eight CTAs collect the sums and tell an eighth of the others alpha, beta and
// whether to go on: a second hop, but the others poll three words instead of a
// thousand (7.2 -> 6.8 us at 400x200).
//
// The set-up is part of the launch: it reads the caller's compact arrays,
// forms the element scales and the first residual (its halo is the first
// exchange), and writes u back in the caller's numbering, so a solve is one or
// two launches instead of ten and one per iteration. All CTAs compute the same
// totals and stop together.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace tpo {

constexpr int RES_ROWS = 30;          // own rows of a group
constexpr int RES_GROUPS = 4;         // groups of a block
constexpr int RES_RED_THREADS = 160;  // threads of the CTA whose summation order is taken over
constexpr int RES_MAX_THREADS = 640;
constexpr int RES_MAX_UNITS = 592;    // groups: their sums lie in shared memory
constexpr int RES_CLUSTER_CTAS = 16;  // non-portable cluster size
constexpr int RES_CLUSTER_GROUPS = 2; // groups of a cluster's CTA at most
constexpr int RES_COPIES = 16;
constexpr int RES_ALL_UNITS = 160, RES_LEADERS = 8;
constexpr int RES_SMEM_MAX = 112 * 1024;  // dynamic: 160 B a thread at most
constexpr int ERR_EXCHANGE_TIMEOUT = 2;

struct ResArgs {
  int nx, ny;
  int L, groups, units, per_cta;  // strip length, row groups, groups of all strips, of a CTA
  double e_min, pen;
  const double *rho, *f;    // caller's arrays, reference numbering
  const uint8_t *fixed;
  double *u;                // warm start in (if warm), solution out
  int warm;
  double tol_sq;
  int max_iter;
  tpo_solve_result *out;    // cluster form, nullable: the asynchronous solve's record
  double *halo[2][2];       // exchanged w: [parity][component], 2 doubles per node
  double *sums;             // exchanged sums: [parity][copy][3][units], 2 doubles each
  double *coef;             // what leaders tell: [parity][leader][3], 2 doubles each
  int leaders;              // CTAs that collect the sums (0: every CTA)
  PcgCtl *ctl;              // out: the end state; err of the cooperative form, zeroed before
  int withhold1;            // failure tests: e + 1 leaves exchange e (0-based) unpublished
};

// two 8-byte elements, each half of v under the epoch
__device__ __forceinline__ void ll_store(double *p, size_t i, double v, uint32_t epoch) {
  const uint64_t x = (uint64_t)__double_as_longlong(v), e = (uint64_t)epoch << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 2 * i),
               "l"(e | (uint32_t)x), "l"(e | x >> 32)
               : "memory");
}
__device__ __forceinline__ bool ll_load(const double *p, size_t i, uint32_t epoch, double &v) {
  uint64_t a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
               : "=l"(a), "=l"(b)
               : "l"(p + 2 * i)
               : "memory");
  v = __longlong_as_double((long long)(b << 32 | (uint32_t)a));
  return a >> 32 == epoch && b >> 32 == epoch;
}

// zero the exchange words and the error word
__global__ void k_res_init(double2 *words, size_t n, PcgCtl *ctl) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    words[i] = make_double2(0.0, 0.0);
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->err = 0;
}

// the asynchronous solve's result record
__device__ __forceinline__ void res_record(int it, int status, int err, double rr, int max_iter,
                                           int launches, tpo_solve_result *out) {
  tpo_solve_result o{};
  o.status = err ? TPO_SOLVE_TIMEOUT : status == TPO_SOLVE_RUNNING ? TPO_SOLVE_MAX_ITER : status;
  o.updates = it;
  o.iters = o.status == TPO_SOLVE_CONVERGED ? it : max_iter;
  o.outer_iters = 1;
  o.rr = rr;
  o.launches = launches;
  *out = o;
}

// a / b for a reciprocal y = RN(1 / b): the quotient RN(a y) corrected twice by
// its exact remainder, which gives the correctly rounded quotient (Markstein,
// IBM J. Res. Dev. 34, 1990) while nothing under- or overflows.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-q, b, a), y, q);
  return fma(fma(-q, b, a), y, q);
}

// Dynamic shared memory of a group (doubles): u of its columns and the forces
// carried into every warp's first column (double2 each), three terms per node
// for the sums, the element scales of the set-up in the terms' space; cluster
// form: w by parity.
__host__ __device__ inline int res_warps(int L) { return (L + 3) / 2; }
__host__ __device__ inline int res_group_doubles(int L, bool cluster) {
  return (cluster ? 10 : 6) * 64 * res_warps(L);
}

template <int PRE, int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 1) k_cgres(ResArgs A) {
  extern __shared__ __align__(16) double res_sm[];
  __shared__ double s_sum[CLUSTER ? 2 : 1][3][CLUSTER ? RES_GROUPS : RES_MAX_UNITS];
  __shared__ double s_red[3][RES_RED_THREADS / 32];
  __shared__ double s_ab[3];  // alpha, beta, 1 if another iteration follows
  const int nx = A.nx, ny = A.ny, ny1 = ny + 1, L = A.L, U = A.units;
  const int W = res_warps(L), C = 2 * W;            // warps, columns of a group
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int cta = blockIdx.x, lg = wid / W, j = wid - lg * W;
  const int unit = cta * A.per_cta + lg, strip = unit / A.groups, grp = unit - strip * A.groups;
  const bool live = unit < U;
  const int gd = res_group_doubles(L, CLUSTER);
  double *um = res_sm + (size_t)lg * gd;
  double2 *su = reinterpret_cast<double2 *>(um);  // [C][32] u
  double2 *sc = su + 32 * C;                      // [W][32] forces carried to column 2 j
  double2 *sw = sc + 32 * W;                      // cluster form: [2][C][32] w
  double *sq = um + (CLUSTER ? 7 : 3) * 32 * C;   // [3][C][32] terms of the sums
  double *se = sq;                                // [C + 1][33] element scales (set-up)

  // this thread's nodes: columns 2 j and 2 j + 1 of the group
  const int x0 = strip * L, x1 = min(x0 + L, nx + 1);
  const int y0 = grp * RES_ROWS - 1, y = y0 + lane;
  const int l1 = min(lane + 1, 31);
  bool in[2], own[2], halo[2], edge[2];
  size_t node[2];
  int h_cta[2] = {0, 0}, h_at[2] = {0, 0};  // cluster form: a halo node's owner, place of its w
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int c = x0 - 1 + 2 * j + e;
    in[e] = live && c >= 0 && c <= min(x1, nx) && y >= 0 && y <= ny;
    own[e] = in[e] && c >= x0 && c < x1 && lane >= 1 && lane <= RES_ROWS;
    halo[e] = in[e] && !own[e];
    edge[e] = own[e] && (c == x0 || c == x1 - 1 || lane == 1 || lane == RES_ROWS);
    node[e] = in[e] ? (size_t)c * ny1 + y : 0;
    if (CLUSTER && halo[e]) {
      const int hu = (c / L) * A.groups + y / RES_ROWS;
      h_cta[e] = hu / A.per_cta;
      h_at[e] = (hu - h_cta[e] * A.per_cta) * (gd / 2) + 32 * (C + W) + (c % L + 1) * 32 +
                y % RES_ROWS + 1;
    }
  }
  auto group_sync = [&]() {  // the threads of this group
    asm volatile("bar.sync %0, %1;" ::"r"(lg + 1), "r"(32 * W) : "memory");
  };

  // ---- element scales: element (x0 - 2 + i, y0 - 1 + k)
  if (live)
    for (int k = j * 32 + lane; k < (C + 1) * 33; k += 32 * W) {
      const int ex = x0 - 2 + k / 33, ey = y0 - 1 + k % 33;
      double v = 0.0;
      if (ex >= 0 && ex < nx && ey >= 0 && ey < ny)
        v = A.e_min + pow(A.rho[(size_t)ex * ny + ey], A.pen) * (1.0 - A.e_min);
      se[k] = v;
    }
  const double2 zero2 = make_double2(0.0, 0.0);
  unsigned m[2] = {0u, 0u};
  double2 x[2] = {zero2, zero2}, r[2] = {zero2, zero2};
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (in[e]) {
      m[e] = A.fixed[node[e]];
      r[e] = reinterpret_cast<const double2 *>(A.f)[node[e]];
      if (A.warm) {
        x[e] = reinterpret_cast<const double2 *>(A.u)[node[e]];
        if (m[e] & FIXED_X) x[e].x = 0.0;
        if (m[e] & FIXED_Y) x[e].y = 0.0;
      }
    }
  __syncthreads();
  double s_el[2] = {0.0, 0.0};  // scales of the elements (c, y) right of the nodes
  double pa[2] = {0.0, 0.0}, pb[2] = {0.0, 0.0}, pd[2] = {0.0, 0.0};  // M^-1
  if (live) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double *q = se + (2 * j + e) * 33 + lane;  // element (c - 1, y - 1)
      s_el[e] = q[34];
      if (in[e]) node_pre<double, PRE>(m[e], q[0], q[1], q[33], q[34], pa[e], pb[e], pd[e]);
    }
  }
  __syncthreads();

  // K v at this thread's own nodes, in the order of the column march: the
  // previous column's elements give fbr + ftr (from below), then the node's
  // column's fbl, then its ftl (from below)
  auto apply = [&](const double2 (&v)[2], double2 (&kv)[2]) {
    if (!live) return;
    su[64 * j + lane] = v[0];
    su[64 * j + 32 + lane] = v[1];
    group_sync();
    const double2 v0u = su[64 * j + l1], v1u = su[64 * j + 32 + l1];
    double2 bl0, br0, tr0, tl0, bl1 = zero2, br1, tr1, tl1 = zero2;
    elem_forces<double>(s_el[0], v[0], v[1], v1u, v0u, bl0, br0, tr0, tl0);
    tl0 = shfl_up2<double>(tl0);
    tr0 = shfl_up2<double>(tr0);
    const double2 carry1 = make_double2(br0.x + tr0.x, br0.y + tr0.y);
    if (j < W - 1) {
      const double2 vr = su[64 * j + 64 + lane], vru = su[64 * j + 64 + l1];
      elem_forces<double>(s_el[1], v[1], vr, vru, v1u, bl1, br1, tr1, tl1);
      tl1 = shfl_up2<double>(tl1);
      tr1 = shfl_up2<double>(tr1);
      sc[32 * j + 32 + lane] = make_double2(br1.x + tr1.x, br1.y + tr1.y);
    }
    group_sync();
    if (own[0]) {
      const double2 carry0 = sc[32 * j + lane];
      kv[0] = make_double2(carry0.x + bl0.x + tl0.x, carry0.y + bl0.y + tl0.y);
      if (m[0] & FIXED_X) kv[0].x = v[0].x;  // identity rows at fixed DOFs
      if (m[0] & FIXED_Y) kv[0].y = v[0].y;
    }
    if (own[1]) {
      kv[1] = make_double2(carry1.x + bl1.x + tl1.x, carry1.y + bl1.y + tl1.y);
      if (m[1] & FIXED_X) kv[1].x = v[1].x;
      if (m[1] & FIXED_Y) kv[1].y = v[1].y;
    }
  };

  // One exchange: publish the edge nodes' `mine` and (with_sums) sum j of the
  // group, held by its warps 0 .. 2; collect the halo nodes' values and all
  // sums in s_sum. False in every thread when a wait ran out (cooperative form).
  const bool lead = CLUSTER || A.leaders == 0 || cta < A.leaders;
  const bool unfilled = !CLUSTER && (cta + 1) * A.per_cta > U;  // the last CTA may have empty groups
  const int copies = A.leaders ? A.leaders : RES_COPIES;
  uint32_t epoch = 0;
  double rz = 0.0, alpha = 0.0, inv_rz = 0.0, inv_alpha = 0.0;
  auto exchange = [&](bool with_sums, double sum, double2 (&mine)[2]) -> bool {
    epoch += 1;
    const int b = epoch & 1;
    const bool publish = CLUSTER || (uint32_t)A.withhold1 != epoch;
    double *sums = A.sums + (size_t)b * 6 * RES_COPIES * U;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (edge[e] && publish) {
        if constexpr (CLUSTER) {
          sw[b * 32 * C + 64 * j + 32 * e + lane] = mine[e];
        } else {
          ll_store(A.halo[b][0], node[e], mine[e].x, epoch);
          ll_store(A.halo[b][1], node[e], mine[e].y, epoch);
        }
      }
    if (with_sums) {
      if (live && j < 3) {
        if constexpr (CLUSTER) {
          if (lane == 0) s_sum[b][j][lg] = sum;
        } else if (lane < copies && publish) {
          ll_store(sums, ((size_t)lane * 3 + j) * U + unit, sum, epoch);
        }
      }
      // while they travel: what beta and p.Kp divide by
      if (wid == 0) {
        inv_rz = 1.0 / (rz + 1e-60);
        inv_alpha = 1.0 / alpha;
      }
    }
    if constexpr (CLUSTER) {
      cluster_sync();
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (halo[e])
          mine[e] = ld_cluster2(reinterpret_cast<double2 *>(res_sm) + h_at[e] + b * 32 * C,
                                h_cta[e]);
      return true;
    } else {
      const int from = cta % copies, words = with_sums ? (lead ? 3 * U : 3) : 0;
      const double *src = lead ? sums + (size_t)from * 6 * U : A.coef + (b * copies + from) * 6;
      double *to = lead ? &s_sum[0][0][0] : s_ab;  // s_sum: [3][units]
      bool need[2] = {halo[0], halo[1]}, ok = true;
      int k = t;  // next word this thread collects
      for (int i = 0; need[0] || need[1] || k < words; ++i) {
        if (k < words) {
          double v;
          if (ll_load(src, k, epoch, v)) {
            to[k] = v;
            k += blockDim.x;
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (need[e]) {
            double2 v;
            const bool hx = ll_load(A.halo[b][0], node[e], epoch, v.x);
            if (ll_load(A.halo[b][1], node[e], epoch, v.y) && hx) {
              mine[e] = v;
              need[e] = false;
            }
          }
        // bounded: some seconds of polls (a load's latency each); another
        // thread's failure ends the wait early
        if ((i & 1023) == 1023) {
          if (*(volatile int *)&A.ctl->err) ok = false;
          if (i >= (1 << 24)) {
            atomicExch(&A.ctl->err, ERR_EXCHANGE_TIMEOUT);
            ok = false;
          }
          if (!ok) break;
        }
      }
      return __syncthreads_and(ok) != 0;
    }
  };

  if (CLUSTER) cluster_sync();  // every CTA has started before another reads its memory

  double2 w[2] = {zero2, zero2}, s[2] = {zero2, zero2}, u[2] = {zero2, zero2},
          p[2] = {zero2, zero2};
  bool ok = true;
  // ---- first residual r = f - K x (zero start: r = f), its halo exchanged
  if (A.warm) {
    double2 kx[2] = {zero2, zero2};
    apply(x, kx);
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (own[e]) {
        r[e].x -= kx[e].x;
        r[e].y -= kx[e].y;
      }
    ok = exchange(false, 0.0, r);
  }

  // ---- iterations; the first pass is the set-up (alpha = beta = 0)
  int it = 0, status = TPO_SOLVE_RUNNING;
  double beta = 0.0, rr = 0.0;
  const double tol_sq = A.tol_sq;
  const int max_iter = A.max_iter;
  // k_cgstep's blocks: thread i of its summing CTA adds blocks i, i + 160, ...;
  // warp w here stands for its warp w
  const int rows = (A.groups + RES_GROUPS - 1) / RES_GROUPS;
  const int NB = (U / A.groups) * rows, nw = (min(NB, RES_RED_THREADS) + 31) / 32;
  auto block_sums = [&](int i, double (&v)[3]) {  // adds those of block i to v
    const int st = i / rows, g0 = (i - st * rows) * RES_GROUPS;
    const int n = min(RES_GROUPS, A.groups - g0), u0 = st * A.groups + g0;
    double pt[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int g = 0; g < RES_GROUPS; ++g)
      if (g < n) {
        const int hc = CLUSTER ? (u0 + g) / A.per_cta : 0, hu = u0 + g - hc * A.per_cta;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double q = CLUSTER ? ld_cluster(&s_sum[epoch & 1][k][hu], hc)
                                   : (&s_sum[0][0][0])[k * U + hu];
          pt[k] = g == 0 ? q : pt[k] + q;
        }
      }
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += pt[k];
  };
  bool init = true;
  while (ok) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (!init) {
        p[e].x = fma(beta, p[e].x, u[e].x);
        p[e].y = fma(beta, p[e].y, u[e].y);
        x[e].x = fma(alpha, p[e].x, x[e].x);
        x[e].y = fma(alpha, p[e].y, x[e].y);
        s[e].x = fma(beta, s[e].x, w[e].x);
        s[e].y = fma(beta, s[e].y, w[e].y);
        r[e].x = fma(-alpha, s[e].x, r[e].x);
        r[e].y = fma(-alpha, s[e].y, r[e].y);
      }
      u[e] = pre_apply<double>(pa[e], pb[e], pd[e], r[e]);
      if (init) p[e] = u[e];
    }
    apply(u, w);
    double sum = 0.0;
    if (live) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        double q0 = 0.0, q1 = 0.0, q2 = 0.0;
        if (own[e]) {
          q0 = node_dot(r[e], u[e]);
          q1 = node_dot(u[e], w[e]);
          q2 = node_sq(r[e]);
        }
        double *q = sq + 64 * j + 32 * e + lane;
        q[0] = q0;
        q[32 * C] = q1;
        q[64 * C] = q2;
      }
      group_sync();
      if (j < 3) {  // sum j of this group: columns in order, then the rows
        const double *q = sq + j * 32 * C + 32 + lane;
        for (int i = 0; i < x1 - x0; i += 8) {
          double v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = i + k < x1 - x0 ? q[32 * (i + k)] : 0.0;
#pragma unroll
          for (int k = 0; k < 8; ++k) sum += v[k];
        }
        sum = warp_sum(sum);
      }
    }
    ok = exchange(true, sum, w);
    if (!ok) break;
    if (lead && wid < nw) {
      double v[3] = {0.0, 0.0, 0.0};
      for (int i = t; i < NB; i += RES_RED_THREADS) block_sums(i, v);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = warp_sum(v[k]);
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) s_red[k][wid] = v[k];
      }
    }
    if (lead) __syncthreads();
    if (lead && wid == 0) {
      double g[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        g[k] = s_red[k][0];
#pragma unroll
        for (int i = 1; i < RES_RED_THREADS / 32; ++i)
          if (i < nw) g[k] += s_red[k][i];
      }
      const double gamma = g[0], delta = g[1];
      rr = g[2];
      double b = 0.0, pap = delta;
      if (!init) {
        b = div_by(gamma, rz + 1e-60, inv_rz);                 // solver.py:151
        pap = delta - div_by(b * gamma, alpha, inv_alpha);     // p_{i+1}.K p_{i+1}
      }
      const double al = gamma / pap;
      const bool fin = finite(gamma) && finite(delta) && finite(rr);
      if (fin && !init) it += 1;
      if (!fin) status = TPO_SOLVE_NONFINITE;
      else if (!init && rr < tol_sq) status = TPO_SOLVE_CONVERGED;  // solver.py:147-149
      else if (!init && it >= max_iter) status = TPO_SOLVE_MAX_ITER;
      else if (fabs(pap) < 1e-30) status = TPO_SOLVE_BREAKDOWN;     // solver.py:114-115
      rz = gamma;
      const double go = status == TPO_SOLVE_RUNNING && it < max_iter ? 1.0 : 0.0;
      if (lane == 0) {
        s_ab[0] = al;
        s_ab[1] = b;
        s_ab[2] = go;
      }
      if (!CLUSTER && A.leaders && lane < 3)
        ll_store(A.coef, ((epoch & 1) * A.leaders + cta) * 3 + lane,
                 lane == 0 ? al : lane == 1 ? b : go, epoch);
    }
    if (lead) __syncthreads();
    alpha = s_ab[0];
    beta = s_ab[1];
    const bool go_on = s_ab[2] != 0.0;
    // In a CTA that does not collect the sums, the next exchange writes s_ab without
    // a barrier. Its groups' own sums hold that back until all their warps have read;
    // an empty group has none. (Two buffers instead cost every CTA 3 % at 400x200.)
    if (!lead && unfilled) __syncthreads();
    if (!go_on) break;
    init = false;
  }
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (own[e] && ok) reinterpret_cast<double2 *>(A.u)[node[e]] = x[e];
  if (cta == 0 && t == 0) {
    A.ctl->it = it;
    A.ctl->rr = rr;
    A.ctl->status = status;
    if (CLUSTER) {
      A.ctl->err = 0;
      if (A.out) res_record(it, status, 0, rr, max_iter, 1, A.out);
    }
  }
  if (CLUSTER) cluster_sync();  // no CTA leaves while another may read its shared memory
}

// the same for the cooperative form, whose waits may have run out in any CTA
__global__ void k_res_result(const PcgCtl *ctl, int max_iter, tpo_solve_result *out) {
  res_record(ctl->it, ctl->status, ctl->err, ctl->rr, max_iter, 3, out);
}

}  // namespace tpo
