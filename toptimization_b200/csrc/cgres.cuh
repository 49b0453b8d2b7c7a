// A whole plain-FP64 solve in one launch, for grids whose PCG state fits on the
// chip: one node per thread, at most one CTA per SM (about 130,000 nodes, 2D,
// point preconditioners); one thread-block cluster where 16 CTAs hold the grid
// (about 10,000 nodes), a cooperative launch otherwise.
//
// On such a grid the one-launch-per-iteration form (k_cgstep) spends 14-16 us
// an iteration on latency: launch, filling the TMA ring, eleven columns one
// after another, and two dependent levels of reduction, while the vectors
// would fit in registers. Here every CTA owns a tile of BX x BY nodes, keeps
// r, s, p, x, u and w of its nodes in registers for the whole solve, and
// exchanges with the other CTAs once per iteration:
//   s = w + beta s, r -= alpha s, u = M^-1 r   on the tile and its halo ring
//   w = K u on the tile, from u in shared memory
//   publish the tile's edge w and its sums gamma, delta, ||r||^2; collect the
//   halo's w and every CTA's sums -> alpha, beta, the stop rules
// The recurrence (Chronopoulos-Gear), the stop rules and their order are those
// of k_cgstep (cgstep.cuh). The halo ring's r and s are kept redundantly, so
// that w is all that crosses between tiles, at the same moment as the sums.
//
// Exchange in a cluster: edge values and sums wait in each CTA's shared memory,
// one cluster barrier, and the readers fetch them from their owners. (Storing
// the sums into every CTA before the barrier: 1.78 instead of 1.75 us an
// iteration at 60x20; storing every warp's, to save the CTA's own reduction: 1.96.)
// Exchange in a cooperative grid, without barriers: a double travels as one 16-byte store of
// {low word, epoch, high word, epoch}; the reader polls its word until both
// epochs are the current exchange's (8-byte accesses are single-copy atomic,
// so data and epoch arrive together). One store and one load latency instead
// of fence + arrive + poll + read. Two buffers by parity of the epoch suffice:
// a CTA publishes exchange e + 2 only after it has every CTA's sums of e + 1,
// which each CTA publishes after it has read all it needs of e. The words are
// zeroed before the launch; epochs start at 1. Every CTA writes its sums to 16
// copies, each polled by a sixteenth of the CTAs: with one copy all CTAs poll
// the same 49 cache lines, and the stores they wait for queue behind the polls
// (5.6 instead of 4.8 us an iteration at 400x200).
//
// The set-up is part of the launch: it reads the caller's compact arrays,
// forms the element scales, the first residual (its halo is the first
// exchange) and writes u back in the caller's numbering, so a solve is one
// memset and one kernel instead of ten launches and one per iteration.
//
// Sums are taken in a fixed order (warp, CTA, then CTAs in order), the same in
// every CTA, so all CTAs stop together and a solve repeats bit by bit.
//
// Measured, per iteration: see res_plan (api.cu).
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace tpo {

struct ResArgs {
  int nx, ny, BX, BY, tiles_y;
  double e_min, pen;
  const double *rho, *f;    // caller's arrays, reference numbering
  const uint8_t *fixed;
  double *u;                // warm start in (if warm), solution out
  int warm;
  double tol_sq;
  int max_iter;
  tpo_solve_result *out;    // cluster form, nullable: the asynchronous solve's record
  double *halo[2][2];       // exchanged w: [parity][component], 2 doubles per node
  double *sums;             // exchanged sums: [parity][copy][3][CTAs], 2 doubles each
  PcgCtl *ctl;              // out: the end state; err of the cooperative form, zeroed before
  int withhold1;            // failure tests: e + 1 leaves exchange e (0-based) unpublished
};

struct LL {
  uint32_t a, b, c, d;
};
__device__ __forceinline__ void ll_store(double *p, size_t i, double v, uint32_t epoch) {
  const uint64_t x = (uint64_t)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(p + 2 * i),
               "r"((uint32_t)x), "r"(epoch), "r"((uint32_t)(x >> 32))
               : "memory");
}
__device__ __forceinline__ bool ll_load(const double *p, size_t i, uint32_t epoch, double &v) {
  LL w;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(w.a), "=r"(w.b), "=r"(w.c), "=r"(w.d)
               : "l"(p + 2 * i)
               : "memory");
  v = __longlong_as_double((long long)(((uint64_t)w.c << 32) | w.a));
  return w.b == epoch && w.d == epoch;
}

// zero the exchange words and the error word
__global__ void k_res_init(double2 *words, size_t n, PcgCtl *ctl) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    words[i] = make_double2(0.0, 0.0);
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->err = 0;
}

// Warp totals of three values with 12 shuffles instead of 30: the halves of
// the warp first split the values between them, then the quarters. Value k's
// total ends in lane 8 k (and its neighbours up to 8 k + 7).
__device__ __forceinline__ double warp_sum3(const double (&v)[3], int lane) {
  const bool hi = lane & 16;
  double a = hi ? v[2] : v[0], b = hi ? 0.0 : v[1];
  a += __shfl_xor_sync(FULL, hi ? v[0] : v[2], 16);
  b += __shfl_xor_sync(FULL, hi ? v[1] : 0.0, 16);
  const bool q = lane & 8;
  double t = q ? b : a;
  t += __shfl_xor_sync(FULL, q ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
  return t;
}

constexpr int RES_MAX_THREADS = 1024;
constexpr int RES_MAX_CTAS = 160;     // cooperative form: five sums per lane of a warp
constexpr int RES_CLUSTER_CTAS = 16;  // non-portable cluster size
constexpr int RES_CLUSTER_THREADS = 768;
constexpr int RES_COPIES = 16;
constexpr int ERR_EXCHANGE_TIMEOUT = 2;

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

// dynamic shared memory: u of the extended tile; cluster form: w of the tile by
// parity; then the element scales of the set-up, whose space the collected
// sums of the cooperative form take over
__host__ __device__ inline size_t res_smem(int BX, int BY, bool cluster) {
  const size_t u = (size_t)(BX + 2) * (BY + 2) * 16;
  const size_t e = (size_t)(BX + 3) * (BY + 3) * 8, q = (size_t)3 * RES_MAX_CTAS * 8;
  return (cluster ? 3 : 1) * u + (e > q ? e : q);
}

template <int PRE, int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 1) k_cgres(ResArgs A) {
  extern __shared__ __align__(16) unsigned char res_sm[];
  __shared__ double red[3 * 32];
  __shared__ double s_mine[2][3];  // cluster form: this CTA's sums, by parity
  __shared__ double s_ab[2];  // alpha, beta
  __shared__ int s_go;        // 1: another iteration
  const int nx = A.nx, ny = A.ny, ny1 = ny + 1;
  const int EY = A.BY + 2, next = (A.BX + 2) * EY;
  double2 *su = reinterpret_cast<double2 *>(res_sm);
  double2 *sw = su + next;  // cluster form only
  double *se = reinterpret_cast<double *>(res_sm + (size_t)next * (CLUSTER ? 48 : 16));
  const int G = gridDim.x, cta = blockIdx.x, t = threadIdx.x, T = blockDim.x;
  const int lane = t & 31, wid = t >> 5, nw = T >> 5;
  const int x0 = (cta / A.tiles_y) * A.BX, y0 = (cta % A.tiles_y) * A.BY;

  // this thread's node: (ix, iy) in the extended tile, (c, y) in the grid
  const int ix = t / EY, iy = t - ix * EY;
  const int c = x0 - 1 + ix, y = y0 - 1 + iy;
  const bool in = t < next && c >= 0 && c <= nx && y >= 0 && y <= ny;
  const bool own = in && ix >= 1 && ix <= A.BX && iy >= 1 && iy <= A.BY;
  const bool halo = in && !own;
  const bool edge = own && (ix == 1 || ix == A.BX || iy == 1 || iy == A.BY);
  const size_t node = in ? (size_t)c * ny1 + y : 0;

  // ---- element scales of the ring: element (x0 - 2 + i, y0 - 2 + j)
  const int SY = A.BY + 3;
  for (int k = t; k < (A.BX + 3) * SY; k += T) {
    const int ex = x0 - 2 + k / SY, ey = y0 - 2 + k % SY;
    double v = 0.0;
    if (ex >= 0 && ex < nx && ey >= 0 && ey < ny)
      v = A.e_min + pow(A.rho[(size_t)ex * ny + ey], A.pen) * (1.0 - A.e_min);
    se[k] = v;
  }
  const unsigned m = in ? A.fixed[node] : 0u;
  double2 x = make_double2(0.0, 0.0);
  if (in && A.warm) {
    x = reinterpret_cast<const double2 *>(A.u)[node];
    if (m & FIXED_X) x.x = 0.0;
    if (m & FIXED_Y) x.y = 0.0;
  }
  double2 r = in ? reinterpret_cast<const double2 *>(A.f)[node] : make_double2(0.0, 0.0);
  if (t < next) su[t] = x;
  __syncthreads();
  NodeScales ns{0.0, 0.0, 0.0, 0.0};
  double pa = 0.0, pb = 0.0, pd = 0.0;
  if (in) {
    const double *q = se + ix * SY + iy;  // element (c-1, y-1)
    ns = NodeScales{q[0], q[1], q[SY], q[SY + 1]};
    node_pre<double, PRE>(m, ns.ll, ns.lh, ns.rl, ns.rh, pa, pb, pd);
  }
  // rows of K at this thread's own node applied to the tile in shared memory
  auto apply = [&](double2 self) {
    const double2 *q = su + t;
    double2 v = node_apply_sym(q[-EY - 1], q[-EY], q[-EY + 1], q[-1], self, q[1], q[EY - 1], q[EY],
                               q[EY + 1], ns);
    if (m & FIXED_X) v.x = self.x;  // identity rows at fixed DOFs
    if (m & FIXED_Y) v.y = self.y;
    return v;
  };

  // cluster form: the halo node's owner and its place in the owner's tile
  int h_cta = 0, h_at = 0;
  if (CLUSTER && halo) {
    const int tx = c / A.BX, ty = y / A.BY;
    h_cta = tx * A.tiles_y + ty;
    h_at = (c - tx * A.BX + 1) * EY + (y - ty * A.BY + 1);
  }

  // One exchange: publish this CTA's sums (v, with_sums) and the edge nodes'
  // `mine`; collect the halo nodes' value and (with_sums), in warp 0, every
  // CTA's sums, lane i those of CTAs i, i + 32, ... added up in v. False in
  // every thread when a wait ran out (cooperative form).
  uint32_t epoch = 0;
  double alpha = 0.0, beta = 0.0, rz = 0.0, inv_rz = 0.0, inv_alpha = 0.0;
  // (set up while the sums travel: the reciprocals the next beta and p.Kp need)
  auto reciprocals = [&]() {
    if (wid == 0) {
      inv_rz = 1.0 / (rz + 1e-60);
      inv_alpha = 1.0 / alpha;
    }
  };
  auto exchange = [&](bool with_sums, double (&v)[3], double2 &mine) -> bool {
    epoch += 1;
    const int b = epoch & 1;
    if constexpr (CLUSTER) {
      if (edge) sw[b * next + t] = mine;
      if (with_sums) {
        const double ws = warp_sum3(v, lane);
        if (lane < 24 && (lane & 7) == 0) red[(lane >> 3) * 32 + wid] = ws;
        __syncthreads();
        if (wid < 3) {
          double w = lane < nw ? red[wid * 32 + lane] : 0.0;
          w = warp_sum(w);
          if (lane == 0) s_mine[b][wid] = w;
        }
      }
      cluster_arrive();
      if (with_sums) reciprocals();
      cluster_wait();
      if (halo) mine = ld_cluster2(sw + b * next + h_at, h_cta);
      if (with_sums && wid == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = lane < G ? ld_cluster(&s_mine[b][k], lane) : 0.0;
      }
      return true;
    }
    const bool publish = (uint32_t)A.withhold1 != epoch;
    if (edge && publish) {
      ll_store(A.halo[b][0], node, mine.x, epoch);
      ll_store(A.halo[b][1], node, mine.y, epoch);
    }
    // [parity][copy][3][CTA]
    double *sums = A.sums + (size_t)b * 6 * RES_COPIES * G;
    if (with_sums) {
      const double ws = warp_sum3(v, lane);
      if (lane < 24 && (lane & 7) == 0) red[(lane >> 3) * 32 + wid] = ws;
      __syncthreads();
      if (wid < 3) {
        double w = lane < nw ? red[wid * 32 + lane] : 0.0;
        w = warp_sum(w);
        if (lane < RES_COPIES && publish)
          ll_store(sums, ((size_t)lane * 3 + wid) * G + cta, w, epoch);
      }
    }
    if (with_sums) reciprocals();
    sums += (size_t)(cta % RES_COPIES) * 6 * G;
    bool need_h = halo, ok = true;
    int k = with_sums ? t : 3 * G;  // next sum this thread collects
    for (int i = 0; need_h || k < 3 * G; ++i) {
      if (k < 3 * G) {
        double w;
        if (ll_load(sums, k, epoch, w)) {
          se[k] = w;
          k += T;
        }
      }
      if (need_h) {
        double2 w;
        const bool hx = ll_load(A.halo[b][0], node, epoch, w.x);
        if (ll_load(A.halo[b][1], node, epoch, w.y) && hx) {
          mine = w;
          need_h = false;
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
    if (!__syncthreads_and(ok)) return false;
    if (with_sums && wid == 0) {
      v[0] = v[1] = v[2] = 0.0;
#pragma unroll
      for (int j = 0; j < RES_MAX_CTAS / 32; ++j) {
        const int i = lane + 32 * j;
        if (i < G) {
          v[0] += se[i];
          v[1] += se[G + i];
          v[2] += se[2 * G + i];
        }
      }
    }
    return true;
  };

  if (CLUSTER) cluster_sync();  // every CTA has started before another reads its memory

  double2 w = make_double2(0.0, 0.0), s = w, u = w, p = w;
  double acc[3] = {0.0, 0.0, 0.0};
  bool ok = true;
  // ---- first residual r = f - K x (zero start: r = f), its halo exchanged
  if (A.warm) {
    if (own) {
      const double2 kx = apply(x);
      r.x -= kx.x;
      r.y -= kx.y;
    }
    ok = exchange(false, acc, r);
  }

  // ---- iterations; the first pass is the set-up (alpha = beta = 0)
  int it = 0, status = TPO_SOLVE_RUNNING;
  double rr = 0.0;
  const double tol_sq = A.tol_sq;
  const int max_iter = A.max_iter;
  bool init = true;
  while (ok) {
    if (!init) {
      p.x = fma(beta, p.x, u.x);
      p.y = fma(beta, p.y, u.y);
      x.x = fma(alpha, p.x, x.x);
      x.y = fma(alpha, p.y, x.y);
      s.x = fma(beta, s.x, w.x);
      s.y = fma(beta, s.y, w.y);
      r.x = fma(-alpha, s.x, r.x);
      r.y = fma(-alpha, s.y, r.y);
    }
    u = pre_apply<double>(pa, pb, pd, r);
    if (init) p = u;
    if (t < next) su[t] = u;
    __syncthreads();
    acc[0] = acc[1] = acc[2] = 0.0;
    if (own) {
      w = apply(u);
      acc[0] = dot2d(r, u);
      acc[1] = dot2d(w, u);
      acc[2] = dot2d(r, r);
    }
    ok = exchange(true, acc, w);
    if (!ok) break;
    if (wid == 0) {
      const double gs = warp_sum3(acc, lane);
      const double gamma = __shfl_sync(FULL, gs, 0), delta = __shfl_sync(FULL, gs, 8);
      rr = __shfl_sync(FULL, gs, 16);
      double b = 0.0, pap = delta;
      if (!init) {
        b = gamma * inv_rz;                    // solver.py:151
        pap = delta - b * gamma * inv_alpha;   // p_{i+1}.K p_{i+1}
      }
      const bool fin = finite(gamma) && finite(delta) && finite(rr);
      if (fin && !init) it += 1;
      if (!fin) status = TPO_SOLVE_NONFINITE;
      else if (!init && rr < tol_sq) status = TPO_SOLVE_CONVERGED;  // solver.py:147-149
      else if (!init && it >= max_iter) status = TPO_SOLVE_MAX_ITER;
      else if (fabs(pap) < 1e-30) status = TPO_SOLVE_BREAKDOWN;     // solver.py:114-115
      rz = gamma;
      if (lane == 0) {
        s_go = status == TPO_SOLVE_RUNNING && it < max_iter;
        s_ab[0] = gamma / pap;
        s_ab[1] = b;
      }
    }
    __syncthreads();
    if (!s_go) break;
    alpha = s_ab[0];
    beta = s_ab[1];
    init = false;
  }
  if (own && ok) reinterpret_cast<double2 *>(A.u)[node] = x;
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
