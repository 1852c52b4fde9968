// cg.cu -- conjugate gradient and power iteration on a plan: the iterative
// callers of the SpMV (no counterpart in the reference, whose programs run one
// SpMV).
//
// One CG iteration is the plan's SpMV q = A p followed by three small kernels:
//   dot   p . q                      (per-CTA partial sums)
//   xr    alpha = rr / sum of the partials;  x += alpha p;  r -= alpha q;
//         partials of r . r
//   p     rr' = sum of the partials; beta = rr' / rr; p = r + beta p
// Every scalar stays on the device, so the iteration is captured once as a
// CUDA graph and replayed; the host reads the residual only every
// `check_every` iterations.  Reductions use a fixed grid and fixed orders, so
// a solve is bit-identical from run to run.  Dot products accumulate in
// double for both FP32 and FP64 vectors.
//
// At 1M unknowns the vectors come from L2, and what counts is launches and loads
// in flight.  So no kernel only adds up partials: each CTA of the next kernel adds
// them itself, all in the same order, while its first vectors are on their way.
// 592 CTAs of 256 threads with two 16-byte loads per vector and thread: as fast with
// one (43.1 to 44.2 us per iteration, FP64, 1024 x 1024 Laplacian), slower with four
// (49.4), with 512 threads (44.7 to 53.2) or 1024 (49.2).  Five
// kernels with scalar loads and one-CTA sums between them: 48.4 us.  Of the 43.6, the
// SpMV takes 27.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <new>

#include "fault.hpp"
#include "internal.hpp"
#include "sparsep.h"

namespace sparsep {
namespace cg {

constexpr int NT = 256;   // threads per CTA of the vector kernels
constexpr int NB = 592;   // CTAs of the vector kernels (4 per SM of a B200)
constexpr int NU = 2;     // vectors of 16 bytes in flight per thread and operand
// sums kept between the kernels: no kernel reads a slot that it writes
enum { S_RR = 0, S_OLD = 1, S_PQ = 2, S_BB = 3, S_QQ = 4, S_NSC = 5 };

// Sum over the CTA, for every thread: lanes, then the warps in order.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sm[NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();  // sm may still be read from the call before
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) s += sm[w];
  return s;
}
__device__ __forceinline__ double partial(const double *__restrict__ part) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NB; i += NT) s += i + threadIdx.x < NB ? part[i + threadIdx.x] : 0.0;
  return s;
}

// 16 bytes of a vector; ALIGNED: all vectors start on 16 bytes
template <typename T> struct alignas(16) Vec {
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};
template <bool ALIGNED, typename T>
__device__ __forceinline__ Vec<T> load(const T *a, size_t i, size_t n) {  // zeros from n on
  constexpr int N = Vec<T>::N;
  Vec<T> r;
  if (ALIGNED && i * N + N <= n) {
    r = reinterpret_cast<const Vec<T> *>(a)[i];
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) r.v[j] = i * N + j < n ? a[i * N + j] : T(0);
  }
  return r;
}
template <bool ALIGNED, typename T>
__device__ __forceinline__ void store(T *a, size_t i, size_t n, const Vec<T> &r) {
  constexpr int N = Vec<T>::N;
  if (ALIGNED && i * N + N <= n) {
    reinterpret_cast<Vec<T> *>(a)[i] = r;
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (i * N + j < n) a[i * N + j] = r.v[j];
  }
}
// f(i0): this thread's vectors i0, i0 + STEP, ... (NU of them, past the end too)
constexpr size_t STEP = (size_t)NB * NT;
template <typename T, typename F>
__device__ __forceinline__ void each(size_t n, F f) {
  const size_t nv = (n + Vec<T>::N - 1) / Vec<T>::N;
  for (size_t i = (size_t)blockIdx.x * NT + threadIdx.x; i < nv; i += NU * STEP) f(i);
}
template <typename T>
__device__ __forceinline__ void add_products(double &s, const Vec<T> &a, const Vec<T> &b) {
#pragma unroll
  for (int j = 0; j < Vec<T>::N; ++j) s += (double)a.v[j] * (double)b.v[j];
}

// part[0, NB): partials of a . b; with BOTH, part[NB, 2 NB): of b . b
template <typename T, bool BOTH, bool ALIGNED>
__global__ void __launch_bounds__(NT, 4) dot(const T *__restrict__ a, const T *__restrict__ b, size_t n,
                                             double *__restrict__ part) {
  double s = 0.0, t = 0.0;
  each<T>(n, [&](size_t i) {
    Vec<T> va[NU], vb[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      va[u] = load<ALIGNED>(a, i + u * STEP, n);
      vb[u] = load<ALIGNED>(b, i + u * STEP, n);
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      add_products(s, va[u], vb[u]);
      if (BOTH) add_products(t, vb[u], vb[u]);
    }
  });
  s = block_sum(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
  if (BOTH) {
    t = block_sum(t);
    if (threadIdx.x == 0) part[NB + blockIdx.x] = t;
  }
}

// sc[s0] and sc[s1]: the sums of the two sets of partials
__global__ void __launch_bounds__(NT) finish(const double *__restrict__ part, double *__restrict__ sc, int s0, int s1) {
  const double a = block_sum(partial(part)), b = block_sum(partial(part + NB));
  if (threadIdx.x == 0) {
    sc[s0] = a;
    sc[s1] = b;
  }
}

// r = b - q; p = r; partials of r . r and b . b
template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(NT, 4) residual(const T *__restrict__ b, const T *__restrict__ q, T *__restrict__ r,
                                                  T *__restrict__ p, size_t n, double *__restrict__ part) {
  double s = 0.0, t = 0.0;
  each<T>(n, [&](size_t i) {
    Vec<T> vb[NU], vq[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      vb[u] = load<ALIGNED>(b, i + u * STEP, n);
      vq[u] = load<ALIGNED>(q, i + u * STEP, n);
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      add_products(t, vb[u], vb[u]);
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j) vq[u].v[j] = vb[u].v[j] - vq[u].v[j];
      add_products(s, vq[u], vq[u]);
      store<ALIGNED>(r, i + u * STEP, n, vq[u]);
      store<ALIGNED>(p, i + u * STEP, n, vq[u]);
    }
  });
  s = block_sum(s);
  t = block_sum(t);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    part[NB + blockIdx.x] = t;
  }
}

// alpha = rr / pq (0 once converged); x += alpha p; r -= alpha q; partials of r . r
template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(NT, 4) update_xr(T *__restrict__ x, T *__restrict__ r, const T *__restrict__ p,
                                                   const T *__restrict__ q, size_t n, double *__restrict__ sc,
                                                   const double *__restrict__ part, double *__restrict__ part_rr) {
  const size_t first = (size_t)blockIdx.x * NT + threadIdx.x;
  const double rr = sc[S_RR], mine = partial(part);
  Vec<T> vr[NU], vq[NU];  // the first ones, under way during the sum
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    vr[u] = load<ALIGNED>(r, first + u * STEP, n);
    vq[u] = load<ALIGNED>(q, first + u * STEP, n);
  }
  const double pq = block_sum(mine);
  const T alpha = (T)(pq != 0.0 ? rr / pq : 0.0);
  double s = 0.0;
  each<T>(n, [&](size_t i) {
    if (i != first) {
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        vr[u] = load<ALIGNED>(r, i + u * STEP, n);
        vq[u] = load<ALIGNED>(q, i + u * STEP, n);
      }
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j)  // past the end nothing counts, whatever alpha is
        vr[u].v[j] = (i + u * STEP) * Vec<T>::N + j < n ? vr[u].v[j] - alpha * vq[u].v[j] : T(0);
      add_products(s, vr[u], vr[u]);
      store<ALIGNED>(r, i + u * STEP, n, vr[u]);
    }
    Vec<T> vx[NU], vp[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      vx[u] = load<ALIGNED>(x, i + u * STEP, n);
      vp[u] = load<ALIGNED>(p, i + u * STEP, n);
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j) vx[u].v[j] += alpha * vp[u].v[j];
      store<ALIGNED>(x, i + u * STEP, n, vx[u]);
    }
  });
  s = block_sum(s);
  if (threadIdx.x == 0) {
    part_rr[blockIdx.x] = s;
    if (blockIdx.x == 0) {
      sc[S_OLD] = rr;
      sc[S_PQ] = pq;
    }
  }
}

// rr' = sum of partials; beta = rr' / rr; p = r + beta p
template <typename T>
__global__ void __launch_bounds__(NT, 4) update_p(T *__restrict__ p, const T *__restrict__ r, size_t n,
                                                  double *__restrict__ sc, const double *__restrict__ part_rr) {
  const size_t first = (size_t)blockIdx.x * NT + threadIdx.x;
  const double old = sc[S_OLD], mine = partial(part_rr);
  Vec<T> vr[NU], vp[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    vr[u] = load<true>(r, first + u * STEP, n);
    vp[u] = load<true>((const T *)p, first + u * STEP, n);
  }
  const double rr = block_sum(mine);
  const T beta = (T)(old != 0.0 ? rr / old : 0.0);
  each<T>(n, [&](size_t i) {
    if (i != first) {
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        vr[u] = load<true>(r, i + u * STEP, n);
        vp[u] = load<true>((const T *)p, i + u * STEP, n);
      }
    }
#pragma unroll
    for (int u = 0; u < NU; ++u) {
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j) vr[u].v[j] += beta * vp[u].v[j];
      store<true>(p, i + u * STEP, n, vr[u]);
    }
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) sc[S_RR] = rr;
}

// power iteration: p = q / ||q|| (p unchanged when q = 0), from the partials of p . q
// and q . q; p and q may be the same vector
template <typename T, bool ALIGNED>
__global__ void __launch_bounds__(NT, 4) normalise(T *p, const T *q, size_t n, double *__restrict__ sc,
                                                   const double *__restrict__ part) {
  const double pq = block_sum(partial(part)), qq = block_sum(partial(part + NB));
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc[S_PQ] = pq;
    sc[S_QQ] = qq;
  }
  if (!(qq > 0.0)) return;
  const T inv = (T)(1.0 / std::sqrt(qq));
  each<T>(n, [&](size_t i) {
    Vec<T> v[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) v[u] = load<ALIGNED>(q, i + u * STEP, n);
#pragma unroll
    for (int u = 0; u < NU; ++u) {
#pragma unroll
      for (int j = 0; j < Vec<T>::N; ++j) v[u].v[j] *= inv;
      store<ALIGNED>(p, i + u * STEP, n, v[u]);
    }
  });
}

}  // namespace cg
}  // namespace sparsep

using namespace sparsep::cg;

struct sparsep_cg {
  sparsep_plan *plan = nullptr;
  int dtype = 0;
  size_t n = 0, esize = 0;
  void *r = nullptr, *p = nullptr, *q = nullptr;
  double *part = nullptr, *sc = nullptr;
  cudaStream_t cap = nullptr;  // capture stream
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  void *graph_x = nullptr;  // x the captured iteration updates
};

static int cg_err(cudaError_t e) {
  if (e == cudaSuccess) return SPARSEP_OK;
  char msg[160];
  std::snprintf(msg, sizeof msg, "%s (%d)", cudaGetErrorString(e), (int)e);
  sparsep::record_error(msg);
  return e == cudaErrorMemoryAllocation ? SPARSEP_ENOMEM : SPARSEP_EIO;
}
#define CGK(x)                               \
  do {                                       \
    cudaError_t e_ = (x);                    \
    if (e_ != cudaSuccess) return cg_err(e_); \
  } while (0)

// The caller's vectors may start on any element: 16-byte accesses only where they can.
static bool on16(const void *a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }

template <typename T>
static int iteration(sparsep_cg *c, T *x, cudaStream_t s) {
  if (int st = sparsep_execute_device(c->plan, c->p, c->q, s)) return st;
  const size_t n = c->n;
  T *r = (T *)c->r, *p = (T *)c->p;
  const T *q = (const T *)c->q;
  double *pq = c->part, *rr = c->part + NB;
  dot<T, false, true><<<NB, NT, 0, s>>>(p, q, n, pq);
  if (on16(x)) update_xr<T, true><<<NB, NT, 0, s>>>(x, r, p, q, n, c->sc, pq, rr);
  else update_xr<T, false><<<NB, NT, 0, s>>>(x, r, p, q, n, c->sc, pq, rr);
  update_p<T><<<NB, NT, 0, s>>>(p, r, n, c->sc, rr);
  return cg_err(cudaGetLastError());
}

template <typename T>
static int solve(sparsep_cg *c, const T *b, T *x, uint32_t max_iters, double tol, uint32_t check_every,
                 uint32_t *iters, double *rel, cudaStream_t s) {
  const size_t n = c->n;
  // r = b - A x; p = r; rr = r.r; bb = b.b
  if (int st = sparsep_execute_device(c->plan, x, c->q, s)) return st;
  if (on16(b)) residual<T, true><<<NB, NT, 0, s>>>(b, (const T *)c->q, (T *)c->r, (T *)c->p, n, c->part);
  else residual<T, false><<<NB, NT, 0, s>>>(b, (const T *)c->q, (T *)c->r, (T *)c->p, n, c->part);
  finish<<<1, NT, 0, s>>>(c->part, c->sc, S_RR, S_BB);
  CGK(cudaGetLastError());
  if (!c->exec || c->graph_x != (void *)x) {
    if (c->exec) cudaGraphExecDestroy(c->exec);
    if (c->graph) cudaGraphDestroy(c->graph);
    c->exec = nullptr;
    c->graph = nullptr;
    CGK(cudaStreamBeginCapture(c->cap, cudaStreamCaptureModeThreadLocal));
    const int st = iteration<T>(c, x, c->cap);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(c->cap, &g);
    if (st) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    CGK(e);
    c->graph = g;
    CGK(cudaGraphInstantiate(&c->exec, c->graph, 0));
    c->graph_x = x;
  }
  double h[S_NSC];
  uint32_t it = 0;
  CGK(cudaMemcpyAsync(h, c->sc, sizeof h, cudaMemcpyDeviceToHost, s));
  CGK(cudaStreamSynchronize(s));
  const double bb = h[S_BB] > 0.0 ? h[S_BB] : 1.0;
  double r = std::sqrt(h[S_RR] / bb);
  const uint32_t every = check_every ? check_every : 1;
  while (r > tol && it < max_iters) {
    const uint32_t k = std::min(every, max_iters - it);
    for (uint32_t j = 0; j < k; ++j) CGK(cudaGraphLaunch(c->exec, s));
    it += k;
    CGK(cudaMemcpyAsync(h, c->sc, sizeof h, cudaMemcpyDeviceToHost, s));
    CGK(cudaStreamSynchronize(s));
    r = std::sqrt(h[S_RR] / bb);
  }
  if (iters) *iters = it;
  if (rel) *rel = r;
  return SPARSEP_OK;
}

// Power iteration: p_0 = x / ||x||; per iteration q = A p, lambda = p . q
// (the Rayleigh quotient, p having unit norm), p = q / ||q||.  The iteration is
// one captured graph (SpMV, both fixed-order dot products, the normalisation);
// the host reads lambda every check_every iterations and stops when two reads
// differ by at most rel_tol * |lambda|.  x receives the last p.
struct sparsep_power {
  sparsep_plan *plan = nullptr;
  int dtype = 0;
  size_t n = 0;
  void *q = nullptr;
  double *part = nullptr, *sc = nullptr;
  cudaStream_t cap = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  void *graph_x = nullptr;
};

// lambda = p . q, p = q / ||q||
template <typename T>
static int power_scale(sparsep_power *w, T *p, const T *q, cudaStream_t s) {
  if (on16(p) && on16(q)) {
    dot<T, true, true><<<NB, NT, 0, s>>>(p, q, w->n, w->part);
    normalise<T, true><<<NB, NT, 0, s>>>(p, q, w->n, w->sc, w->part);
  } else {
    dot<T, true, false><<<NB, NT, 0, s>>>(p, q, w->n, w->part);
    normalise<T, false><<<NB, NT, 0, s>>>(p, q, w->n, w->sc, w->part);
  }
  return cg_err(cudaGetLastError());
}

template <typename T>
static int power_step(sparsep_power *w, T *p, cudaStream_t s) {
  if (int st = sparsep_execute_device(w->plan, p, w->q, s)) return st;
  return power_scale<T>(w, p, static_cast<const T *>(w->q), s);
}

template <typename T>
static int power_run(sparsep_power *w, T *x, uint32_t max_iters, double tol, uint32_t check_every, double *lambda,
                     uint32_t *iters, cudaStream_t s) {
  // p_0 = x / ||x||, in place
  if (int st = power_scale<T>(w, x, x, s)) return st;
  if (!w->exec || w->graph_x != (void *)x) {
    if (w->exec) cudaGraphExecDestroy(w->exec);
    if (w->graph) cudaGraphDestroy(w->graph);
    w->exec = nullptr;
    w->graph = nullptr;
    CGK(cudaStreamBeginCapture(w->cap, cudaStreamCaptureModeThreadLocal));
    const int st = power_step<T>(w, x, w->cap);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(w->cap, &g);
    if (st) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    CGK(e);
    w->graph = g;
    CGK(cudaGraphInstantiate(&w->exec, w->graph, 0));
    w->graph_x = x;
  }
  double h[S_NSC];
  uint32_t it = 0;
  double prev = 0.0, lam = 0.0;
  bool have_prev = false;
  const uint32_t every = check_every ? check_every : 1;
  while (it < max_iters) {
    const uint32_t k = std::min(every, max_iters - it);
    for (uint32_t j = 0; j < k; ++j) CGK(cudaGraphLaunch(w->exec, s));
    it += k;
    CGK(cudaMemcpyAsync(h, w->sc, sizeof h, cudaMemcpyDeviceToHost, s));
    CGK(cudaStreamSynchronize(s));
    lam = h[S_PQ];
    if (!(h[S_QQ] > 0.0)) break;  // A p = 0: lambda = 0 and nothing left to iterate
    if (have_prev && std::fabs(lam - prev) <= tol * std::fabs(lam)) break;
    prev = lam;
    have_prev = true;
  }
  if (lambda) *lambda = lam;
  if (iters) *iters = it;
  return SPARSEP_OK;
}

extern "C" {

int sparsep_cg_create(sparsep_plan *plan, sparsep_cg **out) {
  if (!plan || !out) return SPARSEP_EINVAL;
  *out = nullptr;
  sparsep_plan_info info;
  if (int st = sparsep_plan_get_info(plan, &info)) return st;
  if (info.nrows != info.ncols) return SPARSEP_EINVAL;
  if (info.dtype != SPARSEP_FP32 && info.dtype != SPARSEP_FP64) return SPARSEP_ENOSYS;
  auto *c = new (std::nothrow) sparsep_cg();
  if (!c) return SPARSEP_ENOMEM;
  c->plan = plan;
  c->dtype = info.dtype;
  c->n = info.nrows;
  c->esize = info.dtype == SPARSEP_FP32 ? 4 : 8;
  const size_t vb = (c->n + 64) * c->esize;
  int st = cg_err(sparsep::dev_malloc((void **)&c->r, vb));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&c->p, vb));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&c->q, vb));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&c->part, sizeof(double) * 2 * NB));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&c->sc, sizeof(double) * S_NSC));
  if (!st) st = cg_err(cudaStreamCreateWithFlags(&c->cap, cudaStreamNonBlocking));
  if (st) {
    sparsep_cg_free(c);
    return st;
  }
  *out = c;
  return SPARSEP_OK;
}

void sparsep_cg_free(sparsep_cg *c) {
  if (!c) return;
  if (c->exec) cudaGraphExecDestroy(c->exec);
  if (c->graph) cudaGraphDestroy(c->graph);
  for (void *d : {c->r, c->p, c->q, (void *)c->part, (void *)c->sc})
    if (d) sparsep::dev_free(d);
  if (c->cap) cudaStreamDestroy(c->cap);
  delete c;
}

int sparsep_cg_solve(sparsep_cg *c, const void *d_b, void *d_x, uint32_t max_iters, double rel_tol,
                     uint32_t check_every, uint32_t *iters, double *rel_residual, void *stream) {
  if (!c || !d_b || !d_x || !(rel_tol >= 0.0)) return SPARSEP_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (c->dtype == SPARSEP_FP32)
    return solve<float>(c, (const float *)d_b, (float *)d_x, max_iters, rel_tol, check_every, iters, rel_residual, s);
  return solve<double>(c, (const double *)d_b, (double *)d_x, max_iters, rel_tol, check_every, iters, rel_residual,
                       s);
}

int sparsep_power_create(sparsep_plan *plan, sparsep_power **out) {
  if (!plan || !out) return SPARSEP_EINVAL;
  *out = nullptr;
  sparsep_plan_info info;
  if (int st = sparsep_plan_get_info(plan, &info)) return st;
  if (info.nrows != info.ncols) return SPARSEP_EINVAL;
  if (info.dtype != SPARSEP_FP32 && info.dtype != SPARSEP_FP64) return SPARSEP_ENOSYS;
  auto *w = new (std::nothrow) sparsep_power();
  if (!w) return SPARSEP_ENOMEM;
  w->plan = plan;
  w->dtype = info.dtype;
  w->n = info.nrows;
  const size_t es = info.dtype == SPARSEP_FP32 ? 4 : 8;
  int st = cg_err(sparsep::dev_malloc((void **)&w->q, (w->n + 64) * es));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&w->part, sizeof(double) * 2 * NB));
  if (!st) st = cg_err(sparsep::dev_malloc((void **)&w->sc, sizeof(double) * S_NSC));
  if (!st) st = cg_err(cudaMemset(w->sc, 0, sizeof(double) * S_NSC));
  if (!st) st = cg_err(cudaStreamCreateWithFlags(&w->cap, cudaStreamNonBlocking));
  if (st) {
    sparsep_power_free(w);
    return st;
  }
  *out = w;
  return SPARSEP_OK;
}

void sparsep_power_free(sparsep_power *w) {
  if (!w) return;
  if (w->exec) cudaGraphExecDestroy(w->exec);
  if (w->graph) cudaGraphDestroy(w->graph);
  for (void *d : {w->q, (void *)w->part, (void *)w->sc})
    if (d) sparsep::dev_free(d);
  if (w->cap) cudaStreamDestroy(w->cap);
  delete w;
}

int sparsep_power_run(sparsep_power *w, void *d_x, uint32_t max_iters, double rel_tol, uint32_t check_every,
                      double *lambda, uint32_t *iters, void *stream) {
  if (!w || !d_x || !(rel_tol >= 0.0)) return SPARSEP_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (w->dtype == SPARSEP_FP32)
    return power_run<float>(w, (float *)d_x, max_iters, rel_tol, check_every, lambda, iters, s);
  return power_run<double>(w, (double *)d_x, max_iters, rel_tol, check_every, lambda, iters, s);
}

}  // extern "C"
