// Shared device helpers: vector types, stiffness constants, deterministic
// grid reductions and the device-resident control blocks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "tpo.h"

namespace tpo {

constexpr unsigned FULL = 0xffffffffu;
constexpr int FIXED_X = 1;  // fixed-mask bits (one byte per node)
constexpr int FIXED_Y = 2;

// ---------------------------------------------------------------- constants
// Q4 element stiffness and the regularised inverse used by the element-block
// preconditioner, row-major 8x8, in both precisions. Indices are compile-time
// constants at every use, so each entry becomes a constant-bank operand.
__constant__ double c_ke[64];
__constant__ float c_ke_f[64];
__constant__ double c_kinv[64];
__constant__ float c_kinv_f[64];

// Square-Q4 structure of Ke: Ke = B0^T D B0 + ch (hx hx^T + hy hy^T), where B0
// is the strain matrix at the element centre and hx, hy the hourglass modes.
// {k11, k12, k33, ch, K00, K01} = {D11/4, D12/4, D33/4, ch, Ke[0][0], Ke[0][1]},
// derived from the uploaded Ke and checked against it entry by entry
// (tpo_set_stiffness). Every diagonal entry of such a Ke equals K00, and the
// x-y entry of corner a's 2x2 block is (-1)^a K01.
__constant__ double c_kst[6];
__constant__ float c_kst_f[6];
template <typename T> __device__ __forceinline__ T kst(int i);
template <> __device__ __forceinline__ double kst<double>(int i) { return c_kst[i]; }
template <> __device__ __forceinline__ float kst<float>(int i) { return c_kst_f[i]; }

template <typename T, bool INV> __device__ __forceinline__ T kmat(int i);
template <> __device__ __forceinline__ double kmat<double, false>(int i) { return c_ke[i]; }
template <> __device__ __forceinline__ float kmat<float, false>(int i) { return c_ke_f[i]; }
template <> __device__ __forceinline__ double kmat<double, true>(int i) { return c_kinv[i]; }
template <> __device__ __forceinline__ float kmat<float, true>(int i) { return c_kinv_f[i]; }

// Start of a kernel of the PCG loop that may be launched while the one before it
// still runs (launch_dep): waits for the end of that kernel and its memory, then
// lets the next one be scheduled as this grid's blocks finish. Every thread comes
// here before its first access to memory, so a kernel that waited stands for all
// that came before it. Returns at once after an ordinary launch.
__device__ __forceinline__ void grid_dep() {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

// ---------------------------------------------------------------- vectors
template <typename T> struct V2T;
template <> struct V2T<double> { typedef double2 type; };
template <> struct V2T<float> { typedef float2 type; };
template <typename T> using V2 = typename V2T<T>::type;

template <typename T> __device__ __forceinline__ V2<T> mk2(T x, T y) {
  V2<T> v;
  v.x = x;
  v.y = y;
  return v;
}
__device__ __forceinline__ double fmaT(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmaT(float a, float b, float c) { return fmaf(a, b, c); }

template <typename T> __device__ __forceinline__ V2<T> ld2(const T *base, size_t node) {
  return reinterpret_cast<const V2<T> *>(base)[node];
}
template <typename T> __device__ __forceinline__ void st2(T *base, size_t node, V2<T> v) {
  reinterpret_cast<V2<T> *>(base)[node] = v;
}
template <typename T> __device__ __forceinline__ V2<T> shfl_up2(V2<T> v) {
  return mk2<T>(__shfl_up_sync(FULL, v.x, 1), __shfl_up_sync(FULL, v.y, 1));
}
template <typename T> __device__ __forceinline__ V2<T> shfl_down2(V2<T> v) {
  return mk2<T>(__shfl_down_sync(FULL, v.x, 1), __shfl_down_sync(FULL, v.y, 1));
}

// FP64 dot of two pairs (products of FP32 values are exact in FP64)
template <typename A, typename B>
__device__ __forceinline__ double dot2d(A a, B b) {
  return fma((double)a.x, (double)b.x, (double)a.y * (double)b.y);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(FULL, v, o));
  return v;
}

// ---------------------------------------------------------------- control
// Device-resident PCG state. Fields are written only by the last CTA of a
// kernel (after every other CTA of that kernel has finished) and read by the
// CTAs of later kernels, so no CTA ever reads a field that is being written.
struct PcgCtl {
  double rz;        // r.z of the current residual
  double alpha;     // step length of the current iteration
  double beta;      // coefficient of the next direction update
  double rr;        // latest ||r||^2
  double pap;       // latest p.Ap
  double alpha_prev;  // step length of the iteration before
  double tol_sq;    // stop when rr < tol_sq
  double rupd2;     // mixed form: replace the residual when rr < rupd2 * rmax2 (0: plain)
  double rmax2;     // mixed form: ||r||^2 at the last FP64 residual evaluation
  int32_t it;       // completed updates
  int32_t status;   // TPO_SOLVE_* (or SOLVE_NEED_UPDATE)
  int32_t max_iter;
  int32_t first;    // 1: the next direction is p = z
  int32_t cont;     // mixed form: 1 after a residual replacement (keep p)
  int32_t err;      // nonzero: a bounded wait ran out (TMA pipeline)
  uint32_t counter; // last-CTA ticket
  int32_t since;    // mixed form: iterations since the last residual replacement
  int32_t phase;    // one-launch iteration: launches done (selects the ping-pong buffers)
};

// Outer refinement state of the mixed-precision solve.
struct OuterCtl {
  double rr;        // true FP64 ||f - K u||^2
  double tol_sq;
  int32_t it;       // residual evaluations so far
  int32_t status;   // TPO_SOLVE_*
  uint32_t counter;
  int32_t max_outer;  // residual evaluations allowed (then TPO_SOLVE_MAX_ITER)
};

// Arrival counter of a cooperative grid's barriers, zeroed before the launch.
struct GridBar {
  uint32_t arrived;
  uint32_t err;  // nonzero: a bounded wait ran out
};

struct SumCtl {
  uint32_t counter;
  int32_t pad;
};

// Block partials + last-CTA grid reduction, deterministic for a fixed grid:
// every CTA stores its NV partials (fixed in-block order), the CTA that
// finishes last re-reads all of them in block order and returns true with
// the grid totals in v[] (in every thread). Slot k is a max instead of a sum
// when bit k of MAXMASK is set. `part` holds NV*nblocks doubles. All threads
// of every CTA must call this (no early returns before it).
template <int NV, unsigned MAXMASK = 0u>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], double *part, uint32_t *counter,
                                            int nb, int bid) {
  __shared__ double sm[NV * 32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#define TPO_RED(k, a, b) (((MAXMASK >> (k)) & 1u) ? fmax((a), (b)) : (a) + (b))
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = ((MAXMASK >> k) & 1u) ? warp_max(v[k]) : warp_sum(v[k]);
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sm[k * 32 + wid] = v[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = sm[k * 32];
      for (int w = 1; w < nw; ++w) t = TPO_RED(k, t, sm[k * 32 + w]);
      part[(size_t)k * nb + bid] = t;
    }
    __threadfence();
    const unsigned ticket = atomicAdd(counter, 1u);
    s_last = (ticket == (unsigned)(nb - 1));
  }
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double t = 0.0;  // identity for sums; maxima here are of non-negative values
    for (int i = threadIdx.x; i < nb; i += blockDim.x) t = TPO_RED(k, t, __ldcg(part + (size_t)k * nb + i));
    v[k] = ((MAXMASK >> k) & 1u) ? warp_max(t) : warp_sum(t);
  }
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sm[k * 32 + wid] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double t = sm[k * 32];
    for (int w = 1; w < nw; ++w) t = TPO_RED(k, t, sm[k * 32 + w]);
    v[k] = t;
  }
#undef TPO_RED
  if (threadIdx.x == 0) *counter = 0u;
  return true;
}
// over the whole launch grid
template <int NV, unsigned MAXMASK = 0u>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], double *part, uint32_t *counter) {
  return grid_reduce<NV, MAXMASK>(v, part, counter, (int)(gridDim.x * gridDim.y),
                                  (int)(blockIdx.y * gridDim.x + blockIdx.x));
}

// r^pen for the 3D sensitivities and the 2D compliance. (The solves' scales and
// 2D dc keep pow: with PCG runs on a 1e9 contrast a change of their last bit
// shows.) Whole exponents 0 to 4 (the usual penalties, and
// their derivatives') are products, at most two roundings (1.5 ulp, pow: 2 ulp)
// and a few instructions where pow takes about 150 and 800 cycles of latency.
__device__ __forceinline__ double simp_pow(double r, double pen) {
  if (pen == 3.0) return r * r * r;
  if (pen == 2.0) return r * r;
  if (pen == 1.0) return r;
  if (pen == 0.0) return 1.0;
  if (pen == 4.0) return (r * r) * (r * r);
  return pow(r, pen);
}

__device__ __forceinline__ bool finite(double x) { return isfinite(x); }

// ---------------------------------------------------------------- co-resident CTAs
// Kernels that iterate on the device synchronise their CTAs in one of two
// ways: a thread-block cluster (its barrier, sums exchanged through
// distributed shared memory) or a cooperative launch (a counter in global
// memory). Both offer the same deterministic all-reduce: every CTA gets the
// totals, summed in CTA order, in its shared memory (valid until the next
// call; nullptr when a bounded wait ran out).

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(uint32_t *p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Waits until the counter reaches `target`; about ten seconds at most, after
// which *err is set and false returned.
__device__ __forceinline__ bool wait_count(const uint32_t *p, uint32_t target, uint32_t *err) {
  for (long long i = 0; i < (1ll << 24); ++i) {
    if (ld_acquire(p) >= target) return true;
    if (i > 64) __nanosleep(64);
    if ((i & 1023) == 1023 && ld_acquire(err)) return false;
  }
  atomicExch(err, 1u);
  return false;
}

// Warp totals of up to eight values with 9 shuffles instead of 5 each: halves,
// quarters and eighths of the warp first split the values between them.
// Value k's total ends in lanes 4 k .. 4 k + 3.
template <int NV> __device__ __forceinline__ double warp_sum_split(const double (&v)[NV], int lane) {
  static_assert(NV <= 8, "eight values at most");
  double a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = k < NV ? v[k] : 0.0;
  const bool h = lane & 16, q = lane & 8, e = lane & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double give = h ? a[k] : a[k + 4], keep = h ? a[k + 4] : a[k];
    a[k] = keep + __shfl_xor_sync(FULL, give, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double give = q ? a[k] : a[k + 2], keep = q ? a[k + 2] : a[k];
    a[k] = keep + __shfl_xor_sync(FULL, give, 8);
  }
  const double give = e ? a[0] : a[1], keep = e ? a[1] : a[0];
  double t = keep + __shfl_xor_sync(FULL, give, 4);
  t += __shfl_xor_sync(FULL, t, 2);
  return t + __shfl_xor_sync(FULL, t, 1);
}

// CTA part of the all-reduce: totals of NV per-thread values over the CTA,
// value k in lane 0 of warp k (blockDim.x >= 32 NV; sm holds NV * 32 doubles).
template <int NV, unsigned MAXMASK>
__device__ __forceinline__ double cta_reduce(const double (&v)[NV], double *sm) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if constexpr (MAXMASK == 0u && NV > 3) {
    const double t = warp_sum_split<NV>(v, lane);
    if ((lane & 3) == 0 && lane < 4 * NV) sm[(lane >> 2) * 32 + wid] = t;
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const double t = ((MAXMASK >> k) & 1u) ? warp_max(v[k]) : warp_sum(v[k]);
      if (lane == 0) sm[k * 32 + wid] = t;
    }
  }
  __syncthreads();
  double t = 0.0;
  if (wid < NV) {
    t = lane < nw ? sm[wid * 32 + lane] : 0.0;
    t = ((MAXMASK >> wid) & 1u) ? warp_max(t) : warp_sum(t);
  }
  return t;
}

constexpr int kClusterCtas = 8;  // portable cluster size

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
__device__ __forceinline__ double ld_cluster(const double *sm, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(sm)), b;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(b) : "memory");
  return v;
}
__device__ __forceinline__ double2 ld_cluster2(const double2 *sm, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(sm)), b;
  double2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(b) : "memory");
  return v;
}

// One cluster of kClusterCtas CTAs.
template <int NVMAX> struct ClusterTeam {
  struct Shared {
    double sm[NVMAX * 32];
    double mine[2][NVMAX];  // this CTA's totals, by parity of the call
    double tot[NVMAX];
  };
  Shared &s;
  int calls = 0;
  __device__ explicit ClusterTeam(Shared &sh) : s(sh) {}
  __device__ int rank() const { return (int)cluster_rank(); }
  __device__ int size() const { return kClusterCtas; }
  template <int NV, unsigned MAXMASK = 0u>
  __device__ const double *reduce(const double (&v)[NV]) {
    const double t = cta_reduce<NV, MAXMASK>(v, s.sm);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, b = calls++ & 1;
    if (wid < NV && lane == 0) s.mine[b][wid] = t;
    cluster_sync();
    if (wid < NV) {
      double x = lane < kClusterCtas ? ld_cluster(&s.mine[b][wid], lane) : 0.0;
      x = ((MAXMASK >> wid) & 1u) ? warp_max(x) : warp_sum(x);
      if (lane == 0) s.tot[wid] = x;
    }
    __syncthreads();
    return s.tot;
  }
  // no CTA leaves while another may still read its shared memory
  __device__ void leave() { cluster_sync(); }
};

// A cooperative launch: part holds 2 * NVMAX * size() doubles.
template <int NVMAX> struct GridTeam {
  struct Shared {
    double sm[NVMAX * 32];
    double tot[NVMAX];
    int ok;
  };
  Shared &s;
  GridBar *bar;
  double *part;
  int calls = 0;
  __device__ GridTeam(Shared &sh, GridBar *b, double *p) : s(sh), bar(b), part(p) {}
  __device__ int rank() const { return (int)blockIdx.x; }
  __device__ int size() const { return (int)gridDim.x; }
  template <int NV, unsigned MAXMASK = 0u>
  __device__ const double *reduce(const double (&v)[NV]) {
    const double t = cta_reduce<NV, MAXMASK>(v, s.sm);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, n = size();
    if (n == 1) {
      if (wid < NV && lane == 0) s.tot[wid] = t;
      __syncthreads();
    } else {
      double *pp = part + (size_t)(calls & 1) * NVMAX * n;
      if (wid < NV && lane == 0) pp[wid * n + rank()] = t;
      __syncthreads();
      if (threadIdx.x == 0) {  // the release covers what the barrier ordered before it
        red_release(&bar->arrived, 1u);
        s.ok = wait_count(&bar->arrived, (uint32_t)(calls + 1) * n, &bar->err) ? 1 : 0;
      }
      __syncthreads();
      if (!s.ok) return nullptr;
      if (wid < NV) {
        double x = 0.0;
        for (int i = lane; i < n; i += 32) {
          const double y = __ldcg(pp + wid * n + i);
          x = ((MAXMASK >> wid) & 1u) ? fmax(x, y) : x + y;
        }
        x = ((MAXMASK >> wid) & 1u) ? warp_max(x) : warp_sum(x);
        if (lane == 0) s.tot[wid] = x;
      }
      __syncthreads();
    }
    ++calls;
    return s.tot;
  }
  __device__ void leave() {}
};

}  // namespace tpo
