// Implicit hillslope/marine diffusion on the B200: (I + dt L_kd) h' = h by conjugate gradients
// preconditioned with one geometric-multigrid V-cycle.
//
// The device implementation behind dt_diff_* (include/deeptime_gpu.h). It solves the system of
// the reference's diffusion::solve with DiffusionSolver::Multigrid (crates/deeptime-core/src/
// surface/diffusion.rs:77-110 and surface/diffusion/multigrid.rs:530-763) with its own kernels:
//
//   k_d_coeffs     the operator (diffusion.rs:532-603): east/south face couplings
//                  0.5 (kd_i + kd_j) dt / dx^2 (x wraps when the raster does; 0 on the last row)
//                  and the diagonal ((((1 + east) + west) + south) + north);
//   k_d_apply      y = A x in the reference's term order (diag, east, wrap, west, wrap, south,
//                  north; diffusion.rs:606-650), fused with p.Ap, b - Ax or the mass sums;
//   multigrid      the levels of multigrid.rs:96-199 (2 x 2 aggregation, coarse couplings SCALE
//                  times the fine faces crossing, mass the sum) built on the device per solve, and
//                  two cycles: the reference's (damped Jacobi, omega 0.8, nu 2, to <= 64 cells,
//                  16 sweeps there; multigrid.rs:243-357, :500-523) and a symmetric multi-colour
//                  Gauss-Seidel V(2,2) to a 16 x 8 coarsest level (colours forward before the
//                  coarse correction, backward after it);
//   CG             multigrid::cg_on's loop (stop on the RMS residual, at most 400 iterations, or
//                  on the relative residual), then the mass put-back so sum x = sum b
//                  (multigrid.rs:736-761).
// The CG loop runs on the device as a CUDA-graph conditional WHILE node, like the flexure solve.
// Precision: FP64 CG with an FP32 cycle (the reference's split), FP64 throughout, or an FP32
// inner CG (FP32 cycle) inside FP64 iterative refinement.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"
#include <cuda_pipeline.h>

namespace dt {

enum { DSITE_PAP = 0, DSITE_UPDATE = 1, DSITE_RZ = 2, DSITE_RESID = 3, DSITE_MASS = 4, DSITE_DOT = 5 };
enum { DSTOP_RUNNING = 0, DSTOP_CONVERGED = 1, DSTOP_BREAKDOWN = 2, DSTOP_CAP = 3, DSTOP_NONFINITE = 4 };

struct DScalars {
  double bb, tol;
  int max_it, rule, n;
  double rz, pap, alpha, beta, rr, rz_new;
  int it, stop, body_runs, started;
  double lost, weight, dot_out;
  unsigned long long cond;
  unsigned int ticket[8];
  // reliable updates (DT_DIFF_MIXED_RELIABLE, the FP32 lane): the FP32 residual is replaced by
  // the FP64 one, and x folded into the FP64 accumulation, whenever rr has fallen below
  // delta2 * maxrr or under the tolerance; gate_it == it marks an iteration that does so
  int reliable, gate_it, replacements;
  double delta2, maxrr, rr_true, bb_true;  // rr_true, bb_true: ||b - A x||^2, the reference ||b||^2, unscaled
  unsigned long long cond_if;              // the loop body's IF node around the replacement, 0 without one
};

__device__ __forceinline__ void dset_cond(DScalars* S, unsigned int v) {
  if (S->cond) cudaGraphSetConditional((cudaGraphConditionalHandle)S->cond, v);
}

__device__ __forceinline__ bool d_converged(const DScalars* S, double rr) {
  if (S->rule == DT_STOP_REL_RESIDUAL) return rr <= S->tol * S->tol * S->bb;
  return rr <= S->tol * S->tol * (double)S->n;  // the reference's RMS rule (multigrid.rs:620)
}

// ---------------------------------------------------------------------------------------------
// The operator (diffusion.rs:532-650).

__global__ void k_d_coeffs(int w, int h, int wrap, const double* __restrict__ kd, double dt_over_dx2, double* __restrict__ east,
                           double* __restrict__ south, double* __restrict__ diag, float* __restrict__ east32,
                           float* __restrict__ south32, float* __restrict__ diag32) {
  size_t n = (size_t)w * h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k % w), j = (int)(k / w);
    const double* krow = kd + (size_t)j * w;
    // east face of cell i and of its west neighbour, each as the reference forms it
    auto face_e = [&](int ii) -> double {
      if (ii + 1 < w) return 0.5 * (krow[ii] + krow[ii + 1]) * dt_over_dx2;
      if (wrap) return 0.5 * (krow[ii] + krow[0]) * dt_over_dx2;
      return 0.0;
    };
    auto face_s = [&](int jj) -> double {
      if (jj + 1 < h) return 0.5 * (kd[(size_t)jj * w + i] + kd[(size_t)(jj + 1) * w + i]) * dt_over_dx2;
      return 0.0;
    };
    double e = face_e(i);
    double west = i > 0 ? face_e(i - 1) : (wrap ? face_e(w - 1) : 0.0);
    double s = face_s(j);
    double north = j > 0 ? face_s(j - 1) : 0.0;
    double g = 1.0 + e + west + s + north;
    east[k] = e;
    south[k] = s;
    diag[k] = g;
    east32[k] = (float)e;
    south32[k] = (float)s;
    diag32[k] = (float)g;
  }
}

// y = A x at cell (i, j): diag, east, (wrap), west, (wrap), south, north (diffusion.rs:614-648).
template <class T>
__device__ __forceinline__ T d_apply_at(int w, int h, bool wrap, const T* __restrict__ east, const T* __restrict__ south,
                                        const T* __restrict__ diag, const T* __restrict__ x, int i, int j) {
  size_t c = (size_t)j * w + i, c0 = (size_t)j * w;
  T o = diag[c] * x[c];
  if (i + 1 < w) o -= east[c] * x[c + 1];
  if (wrap && i == w - 1) o -= east[c] * x[c0];
  if (i > 0) o -= east[c - 1] * x[c - 1];
  if (wrap && i == 0) o -= east[c0 + w - 1] * x[c0 + w - 1];
  if (j + 1 < h) o -= south[c] * x[c + w];
  if (j > 0) o -= south[c - w] * x[c - w];
  return o;
}

enum { DA_PAP = 0, DA_RESID = 1, DA_MASS = 2, DA_PLAIN = 3, DA_RESID_GATED = 4 };

// 16 bytes of T, for whole-word loads and stores of a row chunk
template <class T>
struct alignas(16) DV16 {
  T a[16 / sizeof(T)];
};
__device__ __forceinline__ bool d_aligned16(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// y = A x on the row chunk of V = 16 / sizeof(T) cells i0 .. i0 + V - 1 of row j (V divides w),
// every cell's terms in d_apply_at's order: 16-byte loads of the chunk's diag, east and x and of
// the rows below and above (south, x), one value each for the neighbours across the chunk's ends
// (the row's other end where x wraps). 32-bit offsets: the raster has fewer than 2^31 cells.
template <class T>
__device__ __forceinline__ void d_apply_chunk(int w, int h, bool wrap, const T* __restrict__ east, const T* __restrict__ south,
                                              const T* __restrict__ diag, const T* __restrict__ x, int i0, int j,
                                              DV16<T>& ax, DV16<T>& xv, DV16<T>& dg) {
  constexpr int V = 16 / sizeof(T);
  using W = DV16<T>;
  const int c0 = j * w, c = c0 + i0;
  dg = *reinterpret_cast<const W*>(diag + c);
  xv = *reinterpret_cast<const W*>(x + c);
  const W ea = *reinterpret_cast<const W*>(east + c);
  T xl = (T)0, el = (T)0, xr = (T)0;
  if (i0 > 0) {
    xl = x[c - 1];
    el = east[c - 1];
  } else if (wrap) {
    xl = x[c0 + w - 1];
    el = east[c0 + w - 1];
  }
  if (i0 + V < w)
    xr = x[c + V];
  else if (wrap)
    xr = x[c0];
  W xs = {}, ss = {}, xn = {}, sn = {};
  if (j + 1 < h) {
    xs = *reinterpret_cast<const W*>(x + c + w);
    ss = *reinterpret_cast<const W*>(south + c);
  }
  if (j > 0) {
    xn = *reinterpret_cast<const W*>(x + c - w);
    sn = *reinterpret_cast<const W*>(south + c - w);
  }
#pragma unroll
  for (int e = 0; e < V; ++e) {
    const int i = i0 + e;
    const T xe = e + 1 < V ? xv.a[e + 1] : xr;  // east neighbour; x[c0] across the seam
    const T xw = e > 0 ? xv.a[e - 1] : xl, ew = e > 0 ? ea.a[e - 1] : el;  // west neighbour and its east face
    T o = dg.a[e] * xv.a[e];
    if (i + 1 < w) o -= ea.a[e] * xe;
    if (wrap && i == w - 1) o -= ea.a[e] * xe;
    if (i > 0) o -= ew * xw;
    if (wrap && i == 0) o -= ew * xw;
    if (j + 1 < h) o -= ss.a[e] * xs.a[e];
    if (j > 0) o -= sn.a[e] * xn.a[e];
    ax.a[e] = o;
  }
}

// DA_PAP: y = A x, reduce x.y; DA_RESID: y = b - A x, ym = (TM) y, reduce y.y;
// DA_MASS: reduce sum (b - A x) and sum (diag - 1); DA_PLAIN: y = A x; DA_RESID_GATED: in an
// iteration that replaces the residual (S->gate_it == S->it), y = b - A x and y.y -> S->rr_true.
template <class T, class TM, int MODE>
__global__ void __launch_bounds__(256) k_d_apply(int w, int h, int wrap, const T* __restrict__ east, const T* __restrict__ south,
                                                 const T* __restrict__ diag, const T* __restrict__ x, const T* __restrict__ b,
                                                 T* __restrict__ y, TM* __restrict__ ym, double* partials, DScalars* S) {
  if (MODE == DA_PAP && S->stop) {
    if (blockIdx.x == 0 && threadIdx.x == 0) dset_cond(S, 0);
    return;
  }
  if (MODE == DA_RESID_GATED && (S->stop || S->gate_it != S->it)) return;
  size_t n = (size_t)w * h;
  Acc<2> acc;
  acc.v[0] = 0.0;
  acc.v[1] = 0.0;
  constexpr int V = 16 / sizeof(T);
  if (w % V == 0 && n < ((size_t)1 << 31) && d_aligned16(east) && d_aligned16(south) && d_aligned16(diag) && d_aligned16(x) &&
      d_aligned16(b) && d_aligned16(y)) {
    // whole rows of 16-byte chunks, fewer than 2^31 cells: each thread a chunk at a time
    const unsigned int chunks = (unsigned int)(w / V), nch = chunks * (unsigned int)h;
    for (unsigned int q = blockIdx.x * blockDim.x + threadIdx.x; q < nch; q += gridDim.x * blockDim.x) {
      const int j = (int)(q / chunks), i0 = (int)(q - (unsigned int)j * chunks) * V;
      const int c = j * w + i0;
      DV16<T> ax, xv, dg;
      d_apply_chunk<T>(w, h, wrap != 0, east, south, diag, x, i0, j, ax, xv, dg);
      DV16<T> bv = {};
      if (MODE == DA_RESID || MODE == DA_RESID_GATED || MODE == DA_MASS) bv = *reinterpret_cast<const DV16<T>*>(b + c);
      DV16<T> out;
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const T a = ax.a[e];
        if (MODE == DA_PAP) {
          out.a[e] = a;
          acc.v[0] += (double)xv.a[e] * (double)a;
        } else if (MODE == DA_RESID) {
          const T r = bv.a[e] - a;
          out.a[e] = r;
          if (ym) ym[c + e] = (TM)r;
          acc.v[0] += (double)r * (double)r;
        } else if (MODE == DA_RESID_GATED) {
          const T r = bv.a[e] - a;
          out.a[e] = r;
          acc.v[0] += (double)r * (double)r;
        } else if (MODE == DA_MASS) {
          acc.v[0] += (double)bv.a[e] - (double)a;
          acc.v[1] += (double)dg.a[e] - 1.0;
        } else {
          out.a[e] = a;
        }
      }
      if (MODE != DA_MASS) *reinterpret_cast<DV16<T>*>(y + c) = out;
    }
  } else {
    // other widths and unaligned arrays: one cell at a time
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
      int i = (int)(k % w), j = (int)(k / w);
      T ax = d_apply_at<T>(w, h, wrap != 0, east, south, diag, x, i, j);
      if (MODE == DA_PAP) {
        y[k] = ax;
        acc.v[0] += (double)x[k] * (double)ax;
      } else if (MODE == DA_RESID) {
        T r = b[k] - ax;
        y[k] = r;
        if (ym) ym[k] = (TM)r;
        acc.v[0] += (double)r * (double)r;
      } else if (MODE == DA_RESID_GATED) {
        T r = b[k] - ax;
        y[k] = r;
        acc.v[0] += (double)r * (double)r;
      } else if (MODE == DA_MASS) {
        acc.v[0] += (double)b[k] - (double)ax;
        acc.v[1] += (double)diag[k] - 1.0;
      } else {
        y[k] = ax;
      }
    }
  }
  if (MODE == DA_PLAIN) return;
  const int kind[2] = {0, 0};
  int site = MODE == DA_PAP ? DSITE_PAP : (MODE == DA_RESID || MODE == DA_RESID_GATED) ? DSITE_RESID : DSITE_MASS;
  if (reduce_partials<2>(acc, kind, partials, &S->ticket[site], gridDim.x) && threadIdx.x == 0) {
    if (MODE == DA_PAP) {
      S->pap = acc.v[0];
      if (!(acc.v[0] > 0.0) || !isfinite(acc.v[0])) {
        S->stop = isfinite(acc.v[0]) ? DSTOP_BREAKDOWN : DSTOP_NONFINITE;
        dset_cond(S, 0);
      } else {
        S->alpha = S->rz / acc.v[0];
      }
    } else if (MODE == DA_RESID) {
      S->rr = acc.v[0];
    } else if (MODE == DA_RESID_GATED) {
      S->rr_true = acc.v[0];
    } else {
      S->lost = acc.v[0];
      S->weight = acc.v[1];
    }
  }
}

// x += alpha p; r -= alpha Ap; rm = (TM) r (unless null: the cycle reads r itself); reduce r.r and
// test the stopping rule. In 16-byte words of T (the handle's buffers are aligned), up to eight blocks
// an SM. Bound by HBM.
template <class T, class TM>
__global__ void __launch_bounds__(256, 8) k_d_update(size_t n, T* __restrict__ x, T* __restrict__ r, TM* __restrict__ rm,
                                                  const T* __restrict__ p, const T* __restrict__ ap, double* partials, DScalars* S) {
  if (S->stop) {
    if (blockIdx.x == 0 && threadIdx.x == 0) dset_cond(S, 0);
    return;
  }
  constexpr int V = 16 / sizeof(T);
  using W = DV16<T>;
  T alpha = (T)S->alpha;
  Acc<1> acc;
  acc.v[0] = 0.0;
  const size_t nv = n / V, t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
#pragma unroll 1
  for (size_t kv = t0; kv < nv; kv += stride) {
    W xx = reinterpret_cast<W*>(x)[kv], rr = reinterpret_cast<W*>(r)[kv];
    const W pp = reinterpret_cast<const W*>(p)[kv], aa = reinterpret_cast<const W*>(ap)[kv];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      xx.a[e] += alpha * pp.a[e];
      rr.a[e] = rr.a[e] - alpha * aa.a[e];
      acc.v[0] += (double)rr.a[e] * (double)rr.a[e];
    }
    reinterpret_cast<W*>(x)[kv] = xx;
    reinterpret_cast<W*>(r)[kv] = rr;
    if (rm) {
#pragma unroll
      for (int e = 0; e < V; ++e) rm[kv * V + e] = (TM)rr.a[e];
    }
  }
  for (size_t k = nv * V + t0; k < n; k += stride) {
    x[k] += alpha * p[k];
    T rv = r[k] - alpha * ap[k];
    r[k] = rv;
    if (rm) rm[k] = (TM)rv;
    acc.v[0] += (double)rv * (double)rv;
  }
  const int kind[1] = {0};
  if (reduce_partials<1>(acc, kind, partials, &S->ticket[DSITE_UPDATE], gridDim.x) && threadIdx.x == 0) {
    double rr = acc.v[0];
    S->rr = rr;
    S->it += 1;
    if (S->reliable) {
      // the FP32 residual only asks for a replacement; the FP64 residual decides convergence
      bool gate = false;
      if (!isfinite(rr)) {
        S->stop = DSTOP_NONFINITE;
      } else if (rr <= S->tol * S->tol * S->bb || rr < S->delta2 * S->maxrr) {
        S->gate_it = S->it;
        gate = true;
      } else if (S->it >= S->max_it) {
        S->stop = DSTOP_CAP;
      }
      if (S->cond_if) cudaGraphSetConditional((cudaGraphConditionalHandle)S->cond_if, gate ? 1u : 0u);
      if (S->stop) dset_cond(S, 0);
      return;
    }
    if (!isfinite(rr))
      S->stop = DSTOP_NONFINITE;
    else if (d_converged(S, rr))
      S->stop = DSTOP_CONVERGED;
    else if (S->it >= S->max_it)
      S->stop = DSTOP_CAP;
    if (S->stop) dset_cond(S, 0);
  }
}

// After the cycle, with rz = r . z: beta = rz / rz_old (multigrid.rs:721-727).
__device__ __forceinline__ void d_finish_rz(DScalars* S, double rz) {
  if (!S->started) {
    S->started = 1;
    S->rz = rz;
    if (!isfinite(rz)) S->stop = DSTOP_NONFINITE;
    return;
  }
  if (!(isfinite(rz) && S->rz > 0.0)) {
    S->stop = isfinite(rz) ? DSTOP_BREAKDOWN : DSTOP_NONFINITE;
    dset_cond(S, 0);
    return;
  }
  S->beta = rz / S->rz;
  S->rz = rz;
}
// rz = r . z, where the finest level's post-smoothing does not form it (k_mg_tile).
template <class T, class TM>
__global__ void __launch_bounds__(256, 8) k_d_rz(size_t n, const T* __restrict__ r, const TM* __restrict__ z, double* partials,
                                              DScalars* S) {
  if (S->stop) return;
  Acc<1> acc;
  acc.v[0] = 0.0;
  constexpr int V = 16 / sizeof(T);
  const size_t nv = n / V, t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
  for (size_t kv = t0; kv < nv; kv += stride) {
    const DV16<T> rr = reinterpret_cast<const DV16<T>*>(r)[kv];
#pragma unroll
    for (int e = 0; e < V; ++e) acc.v[0] += (double)rr.a[e] * (double)z[kv * V + e];
  }
  for (size_t k = nv * V + t0; k < n; k += stride) acc.v[0] += (double)r[k] * (double)z[k];
  const int kind[1] = {0};
  if (reduce_partials<1>(acc, kind, partials, &S->ticket[DSITE_RZ], gridDim.x) && threadIdx.x == 0) {
    d_finish_rz(S, acc.v[0]);
  }
}

// p = z + beta p (p = z on the first direction), and the loop guard.
template <class T, class TM>
__global__ void __launch_bounds__(256, 8) k_d_direction(size_t n, T* __restrict__ p, const TM* __restrict__ z, DScalars* S, int first) {
  if (!first && blockIdx.x == 0 && threadIdx.x == 0) {
    int runs = ++S->body_runs;
    bool again = S->stop == 0 && runs < S->max_it + 2;
    if (!again && S->stop == 0) S->stop = DSTOP_CAP;
    dset_cond(S, again ? 1u : 0u);
  }
  if (S->stop) return;
  T beta = first ? (T)0 : (T)S->beta;
  constexpr int V = 16 / sizeof(T);
  using W = DV16<T>;
  const size_t nv = n / V, t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
#pragma unroll 1
  for (size_t kv = t0; kv < nv; kv += stride) {
    W pp;
    if (!first) pp = reinterpret_cast<const W*>(p)[kv];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const T zz = (T)z[kv * V + e];
      pp.a[e] = first ? zz : zz + beta * pp.a[e];
    }
    reinterpret_cast<W*>(p)[kv] = pp;
  }
  for (size_t k = nv * V + t0; k < n; k += stride) p[k] = first ? (T)z[k] : (T)z[k] + beta * p[k];
}

// ---------------------------------------------------------------------------------------------
// The multigrid levels (multigrid.rs:96-199).

template <class TM>
struct DLevel {
  int w, h, wrap;
  TM *east, *south, *diag, *wd, *mass, *r, *z, *t;
};

// The finest level's wd = omega / diag; its other coefficients are the operator's own arrays.
template <class TM>
__global__ void k_mg_finest(size_t n, const TM* __restrict__ diag, TM omega, TM* __restrict__ wd) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) wd[k] = omega / diag[k];
}

// Coarse mass and faces: mass = sum of the 2 x 2 block's; east = SCALE * the fine east faces
// leaving its last column (wrapping), south = SCALE * the fine south faces of its last row.
template <class TM>
__global__ void k_mg_coarsen(DLevel<TM> f, DLevel<TM> c, TM scale) {
  size_t nc = (size_t)c.w * c.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nc; k += (size_t)gridDim.x * blockDim.x) {
    int ic = (int)(k % c.w), jc = (int)(k / c.w);
    int r0 = 2 * jc, r1 = min(2 * jc + 2, f.h), c0 = 2 * ic, c1 = min(2 * ic + 2, f.w);
    int last_row = r1 - 1, last_col = c1 - 1;
    TM m = 0;
    for (int j = r0; j < r1; ++j)
      for (int i = c0; i < c1; ++i) m += f.mass ? f.mass[(size_t)j * f.w + i] : (TM)1;
    c.mass[k] = m;
    TM e = 0;
    if (ic + 1 < c.w || c.wrap) {
      for (int j = r0; j < r1; ++j) e += f.east[(size_t)j * f.w + last_col];
      e = scale * e;
    }
    c.east[k] = e;
    TM s = 0;
    if (jc + 1 < c.h) {
      for (int i = c0; i < c1; ++i) s += f.south[(size_t)last_row * f.w + i];
      s = scale * s;
    }
    c.south[k] = s;
  }
}

template <class TM>
__global__ void k_mg_diag(DLevel<TM> c, TM omega) {
  size_t nc = (size_t)c.w * c.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nc; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k % c.w), j = (int)(k / c.w);
    size_t c0 = (size_t)j * c.w;
    TM west = i > 0 ? c.east[k - 1] : (c.wrap ? c.east[c0 + c.w - 1] : (TM)0);
    TM north = j > 0 ? c.south[k - c.w] : (TM)0;
    TM g = c.mass[k] + c.east[k] + west + c.south[k] + north;
    c.diag[k] = g;
    c.wd[k] = omega / g;
  }
}

// Products rounded on their own (never fused into an add): the cycle's kernels form the same
// values whichever kernel runs them, as the reference forms them (no fused multiply-adds).
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }

// A z at a cell of a level, in the level's term order (multigrid.rs:202-240), reading z (+ the
// coarse correction of each cell's parent when zc is given).
template <class TM>
__device__ __forceinline__ TM mg_apply_at(const DLevel<TM>& L, const TM* __restrict__ z, const TM* __restrict__ zc, int wc, int i,
                                          int j) {
  auto zat = [&](int ii, int jj) -> TM {
    TM v = z[(size_t)jj * L.w + ii];
    if (zc) v += zc[(size_t)(jj / 2) * wc + ii / 2];
    return v;
  };
  size_t c = (size_t)j * L.w + i, c0 = (size_t)j * L.w;
  TM o = mulr(L.diag[c], zat(i, j));
  if (i + 1 < L.w) o -= mulr(L.east[c], zat(i + 1, j));
  if (i > 0) o -= mulr(L.east[c - 1], zat(i - 1, j));
  if (L.wrap) {
    if (i == L.w - 1) o -= mulr(L.east[c], zat(0, j));
    if (i == 0) o -= mulr(L.east[c0 + L.w - 1], zat(L.w - 1, j));
  }
  if (j + 1 < L.h) o -= mulr(L.south[c], zat(i, j + 1));
  if (j > 0) o -= mulr(L.south[c - L.w], zat(i, j - 1));
  return o;
}

// z = wd r (the first sweep from z = 0)
template <class TM>
__global__ void k_mg_first(DLevel<TM> L, TM* __restrict__ z) {
  size_t n = (size_t)L.w * L.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) z[k] = L.wd[k] * L.r[k];
}

// zout = z' + wd (r - A z'), z' = zin (+ the coarse correction)
template <class TM>
__global__ void k_mg_sweep(DLevel<TM> L, const TM* __restrict__ zin, TM* __restrict__ zout, const TM* __restrict__ zc, int wc) {
  size_t n = (size_t)L.w * L.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k % L.w), j = (int)(k / L.w);
    TM zk = zin[k];
    if (zc) zk += zc[(size_t)(j / 2) * wc + i / 2];
    TM az = mg_apply_at<TM>(L, zin, zc, wc, i, j);
    zout[k] = zk + L.wd[k] * (L.r[k] - az);
  }
}

// rc = sum over each 2 x 2 block of (r - A z) (multigrid.rs:332-356)
template <class TM, class K>
__device__ __forceinline__ void restrict_cell(const DLevel<TM>& L, const TM* __restrict__ z, const DLevel<TM>& C, K k) {
  int ic = (int)(k % C.w), jc = (int)(k / C.w);
  TM acc = 0;
  for (int j = 2 * jc; j < min(2 * jc + 2, L.h); ++j)
    for (int i = 2 * ic; i < min(2 * ic + 2, L.w); ++i) acc += L.r[(size_t)j * L.w + i] - mg_apply_at<TM>(L, z, nullptr, 0, i, j);
  C.r[k] = acc;
}
template <class TM>
__global__ void k_mg_restrict(DLevel<TM> L, const TM* __restrict__ z, DLevel<TM> C) {
  size_t nc = (size_t)C.w * C.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nc; k += (size_t)gridDim.x * blockDim.x)
    restrict_cell<TM>(L, z, C, k);
}

// The colour of a cell for the Gauss-Seidel sweeps: (i + j) % 2, and on a wrapping level of odd
// width the last column takes two colours of its own (2 + j % 2), since a ring of odd length has
// no two-colouring. No two cells of one colour are neighbours.
__device__ __forceinline__ int gs_colour(int w, int wrap, int i, int j) {
  if (wrap && (w & 1) && i == w - 1) return 2 + (j & 1);
  return (i + j) & 1;
}
inline int gs_colours(int w, int wrap) { return (wrap && (w & 1)) ? 4 : 2; }

// One Gauss-Seidel update of cell k = (i, j) of colour `colour`: z_c += (r - A z)_c / diag_c.
// FIRST: z is taken as 0 where this sweep has not written (the cycle's first sweep).
template <class TM, bool FIRST>
__device__ __forceinline__ void gs_cell_at(const DLevel<TM>& L, TM* __restrict__ z, int colour, size_t k, int i, int j) {
  // in the first forward sweep, cells of later colours still hold 0 (not yet written)
  auto zat = [&](int ii, int jj) -> TM {
    if (FIRST && gs_colour(L.w, L.wrap, ii, jj) >= colour) return (TM)0;
    return z[(size_t)jj * L.w + ii];
  };
  size_t c = k, c0 = (size_t)j * L.w;
  TM zk = FIRST ? (TM)0 : z[c];
  TM o = mulr(L.diag[c], zk);
  if (i + 1 < L.w) o -= mulr(L.east[c], zat(i + 1, j));
  if (i > 0) o -= mulr(L.east[c - 1], zat(i - 1, j));
  if (L.wrap) {
    if (i == L.w - 1) o -= mulr(L.east[c], zat(0, j));
    if (i == 0) o -= mulr(L.east[c0 + L.w - 1], zat(L.w - 1, j));
  }
  if (j + 1 < L.h) o -= mulr(L.south[c], zat(i, j + 1));
  if (j > 0) o -= mulr(L.south[c - L.w], zat(i, j - 1));
  z[c] = zk + mulr(L.r[c] - o, L.wd[c]);  // wd = 1 / diag on the Gauss-Seidel hierarchy
}
template <class TM, bool FIRST>
__device__ __forceinline__ void gs_cell(const DLevel<TM>& L, TM* __restrict__ z, int colour, size_t k) {
  gs_cell_at<TM, FIRST>(L, z, colour, k, (int)(k % L.w), (int)(k / L.w));
}

// One Gauss-Seidel pass over the cells of colour `colour`.
template <class TM, bool FIRST>
__global__ void k_mg_gs(DLevel<TM> L, TM* __restrict__ z, int colour) {
  size_t n = (size_t)L.w * L.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k % L.w), j = (int)(k / L.w);
    if (gs_colour(L.w, L.wrap, i, j) != colour) continue;
    gs_cell<TM, FIRST>(L, z, colour, k);
  }
}

// z += P zc (piecewise constant)
template <class TM>
__global__ void k_mg_prolong(DLevel<TM> L, TM* __restrict__ z, const TM* __restrict__ zc, int wc) {
  size_t n = (size_t)L.w * L.h;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k % L.w), j = (int)(k / L.w);
    z[k] += zc[(size_t)(j / 2) * wc + i / 2];
  }
}

// The coarsest level in one block (at most 128 cells): KIND 0 the reference's first sweep and
// 15 damped Jacobi sweeps (multigrid.rs:504-512); KIND 1 eight forward and eight backward
// multi-colour Gauss-Seidel sweeps. Result in z. Every thread of the block takes part.
template <class TM, int KIND>
__device__ __forceinline__ void coarsest_solve(const DLevel<TM>& L, TM* __restrict__ z, int sweeps) {
  __shared__ TM sz[2][256];
  int n = L.w * L.h;
  int k = threadIdx.x;
  if (KIND == 0) {
    if (k < n) sz[0][k] = L.wd[k] * L.r[k];
    __syncthreads();
    int cur = 0;
    for (int s = 1; s < sweeps; ++s) {
      if (k < n) {
        int i = k % L.w, j = k / L.w;
        TM az = mg_apply_at<TM>(L, sz[cur], nullptr, 0, i, j);
        sz[cur ^ 1][k] = sz[cur][k] + L.wd[k] * (L.r[k] - az);
      }
      __syncthreads();
      cur ^= 1;
    }
    if (k < n) z[k] = sz[cur][k];
  } else {
    if (k < n) sz[0][k] = (TM)0;
    __syncthreads();
    int ncol = (L.wrap && (L.w & 1)) ? 4 : 2;
    for (int pass = 0; pass < 2 * sweeps; ++pass) {
      bool forward = pass < sweeps;
      for (int q = 0; q < ncol; ++q) {
        int colour = forward ? q : ncol - 1 - q;
        if (k < n) {
          int i = k % L.w, j = k / L.w;
          if (gs_colour(L.w, L.wrap, i, j) == colour) {
            TM az = mg_apply_at<TM>(L, sz[0], nullptr, 0, i, j);
            sz[0][k] = sz[0][k] + mulr(L.r[k] - az, L.wd[k]);
          }
        }
        __syncthreads();
      }
    }
    if (k < n) z[k] = sz[0][k];
  }
}
template <class TM, int KIND>
__global__ void k_mg_coarsest(DLevel<TM> L, TM* __restrict__ z, int sweeps) {
  coarsest_solve<TM, KIND>(L, z, sweeps);
}

// The V-cycle's part from a level of at most MG_BLOCK_CELLS cells down, in one block: the separate
// launches' passes in their order (pre-sweeps, restriction, the coarser levels, coarse correction,
// post-sweeps; the coarsest level's sweeps), so the same values. The levels' arrays are staged in
// shared memory (off[q]: the level's first cell there, seven arrays of `total` cells). Bound by the
// latency of some 35 to 60 dependent passes, so a thread keeps its cells' couplings and neighbours'
// places in registers through a level's passes, and a level's barriers take only the warps that hold
// its cells (barrier q + 1; the others wait where they meet the level again on the way up). With the
// indexes worked out in every pass and all 1024 threads in every barrier a Gauss-Seidel chain from
// 64 x 32 cells took 29 us and a Jacobi one from 64 x 21 21.6 us; this 18.7 and
// 14.4 (cold caches).
constexpr int MG_BLOCK_LEVELS = 8;
constexpr int MG_BLOCK_CELLS = 2048;  // two cells a thread
template <class TM>
struct MgChain {
  DLevel<TM> lv[MG_BLOCK_LEVELS];
  int off[MG_BLOCK_LEVELS];
  int count, total;
};
// One cell of a staged level: couplings (0 where there is no neighbour, whose place is then the
// cell's own), in mg_apply_at's order of terms (`seam`: the west term before the east one).
template <class TM>
struct MgCell {
  TM d, wd, r, e, w, s, n;
  int k, ke, kw, ks, kn, colour;
  bool seam;
  __device__ __forceinline__ TM apply(const TM* z) const {
    TM o = mulr(d, z[k]);
    const TM a = mulr(e, z[ke]), b = mulr(w, z[kw]);
    o -= seam ? b : a;
    o -= seam ? a : b;
    o -= mulr(s, z[ks]);
    o -= mulr(n, z[kn]);
    return o;
  }
};
template <class TM, bool JAC>
__global__ void __launch_bounds__(1024) k_mg_coarse(MgChain<TM> g, int nu, int coarse_sweeps) {
  const int tid = threadIdx.x, nt = blockDim.x;
  extern __shared__ __align__(16) unsigned char mg_chain_smem[];
  TM* const sbase = reinterpret_cast<TM*>(mg_chain_smem);
  // arrays of a level: 0 z, 1 t (Jacobi's other buffer; the residuals), 2 r, 3 diag, 4 wd, 5 east, 6 south
  auto arr = [&](int a, int q) { return sbase + a * g.total + g.off[q]; };
  for (int q = 0; q < g.count; ++q) {
    const DLevel<TM>& G = g.lv[q];
    for (int k = tid; k < G.w * G.h; k += nt) {
      arr(0, q)[k] = (TM)0;
      if (q == 0) __pipeline_memcpy_async(arr(2, q) + k, G.r + k, sizeof(TM));
      __pipeline_memcpy_async(arr(3, q) + k, G.diag + k, sizeof(TM));
      __pipeline_memcpy_async(arr(4, q) + k, G.wd + k, sizeof(TM));
      __pipeline_memcpy_async(arr(5, q) + k, G.east + k, sizeof(TM));
      __pipeline_memcpy_async(arr(6, q) + k, G.south + k, sizeof(TM));
    }
  }
  __pipeline_commit();
  __pipeline_wait_prior(0);
  __syncthreads();
  auto cells = [&](int q) { return g.lv[q].w * g.lv[q].h; };
  auto threads = [&](int q) { return min(nt, (cells(q) + 31) & ~31); };
  auto bar = [&](int q) { asm volatile("bar.sync %0, %1;" ::"r"(q + 1), "r"(threads(q)) : "memory"); };
  MgCell<TM> cell[2];
  bool has[2];
  auto load = [&](int q) {
    const int w = g.lv[q].w, h = g.lv[q].h, wrap = g.lv[q].wrap;
    const TM *east = arr(5, q), *south = arr(6, q);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = tid + u * nt;
      has[u] = k < w * h;
      if (!has[u]) continue;
      const int j = k / w, i = k - j * w;
      MgCell<TM>& c = cell[u];
      c.k = k;
      c.d = arr(3, q)[k];
      c.wd = arr(4, q)[k];
      c.r = arr(2, q)[k];
      const bool he = i + 1 < w || wrap, hw = i > 0 || wrap;
      c.ke = i + 1 < w ? k + 1 : wrap ? j * w : k;
      c.kw = i > 0 ? k - 1 : wrap ? k + w - 1 : k;
      c.ks = j + 1 < h ? k + w : k;
      c.kn = j > 0 ? k - w : k;
      c.e = he ? east[k] : (TM)0;
      c.w = hw ? east[c.kw] : (TM)0;
      c.s = j + 1 < h ? south[k] : (TM)0;
      c.n = j > 0 ? south[k - w] : (TM)0;
      c.seam = wrap && i == w - 1;
      c.colour = gs_colour(w, wrap, i, j);
    }
  };
  // `count` sweeps of level q on its current z (in buffer `cur`, 0 z or 1 t; Gauss-Seidel: z in place,
  // colours up when `forward`); the buffer that holds the result
  auto sweeps = [&](int q, int cur, int count, bool forward) {
    if constexpr (JAC) {
      for (int sw = 0; sw < count; ++sw, cur ^= 1) {
        const TM* zi = arr(cur, q);
        TM* zo = arr(cur ^ 1, q);
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (has[u]) {
            const TM zk = zi[cell[u].k];
            zo[cell[u].k] = zk + cell[u].wd * (cell[u].r - cell[u].apply(zi));
          }
        bar(q);
      }
    } else {
      const int ncol = (g.lv[q].wrap && (g.lv[q].w & 1)) ? 4 : 2;
      TM* z = arr(0, q);
      for (int sw = 0; sw < count; ++sw)
        for (int p = 0; p < ncol; ++p) {
          const int colour = forward ? p : ncol - 1 - p;
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (has[u] && cell[u].colour == colour) z[cell[u].k] += mulr(cell[u].r - cell[u].apply(z), cell[u].wd);
          bar(q);
        }
    }
    return cur;
  };
  // z = wd r, Jacobi's first sweep
  auto first = [&](int q) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (has[u]) arr(0, q)[cell[u].k] = cell[u].wd * cell[u].r;
    bar(q);
  };
  // a Jacobi level's z is in buffer `down` after its nu sweeps down (the first in z)
  const int last = g.count - 1, down = JAC ? (nu - 1) & 1 : 0;
  int q = 0;
  for (; tid < threads(q); ++q) {
    load(q);
    if (q > 0) {
      // r: the sum over the block of 2 x 2 finer cells of their residuals
      const int w = g.lv[q].w, wf = g.lv[q - 1].w, hf = g.lv[q - 1].h;
      const TM* res = arr(down ^ 1, q - 1);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (has[u]) {
          const int jc = cell[u].k / w, ic = cell[u].k - jc * w;
          TM acc = 0;
          for (int j = 2 * jc; j < min(2 * jc + 2, hf); ++j)
            for (int i = 2 * ic; i < min(2 * ic + 2, wf); ++i) acc += res[j * wf + i];
          cell[u].r = acc;
          arr(2, q)[cell[u].k] = acc;
        }
    }
    if (JAC) first(q);
    if (q == last) break;
    if (JAC)
      sweeps(q, 0, nu - 1, true);
    else
      sweeps(q, 0, nu, true);
    // the residuals into the buffer that does not hold z
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (has[u]) arr(down ^ 1, q)[cell[u].k] = cell[u].r - cell[u].apply(arr(down, q));
    bar(q);
  }
  int top = down;  // the buffer of the finest level's result
  if (q == last && tid < threads(last)) {
    int cur;
    if (JAC) {
      cur = sweeps(last, 0, coarse_sweeps - 1, true);
    } else {
      sweeps(last, 0, coarse_sweeps, true);
      cur = sweeps(last, 0, coarse_sweeps, false);
    }
    if (last == 0) top = cur;
    // the level above reads the result from z
    if (last > 0 && cur == 1) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (has[u]) arr(0, last)[cell[u].k] = arr(1, last)[cell[u].k];
    }
  }
  // where a level's result lies on the way up: nu sweeps from `down`
  const int up = JAC ? (down + nu) & 1 : 0;
  for (q = min(q, g.count) - 1; q >= 0; --q) {
    bar(q);  // the coarser level's result is there
    load(q);
    const int wc = g.lv[q + 1].w, w = g.lv[q].w;
    const TM* zc = arr(q + 1 == last ? 0 : up, q + 1);
    TM* z = arr(down, q);
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (has[u]) {
        const int j = cell[u].k / w, i = cell[u].k - j * w;
        z[cell[u].k] += zc[(j / 2) * wc + i / 2];
      }
    bar(q);
    top = sweeps(q, down, nu, false);
  }
  if (tid < threads(0)) {
    // every thread of the finest level wrote its own cells
    for (int k = tid; k < cells(0); k += nt) g.lv[0].z[k] = arr(top, 0)[k];
  }
}

// A level's smoothing in one launch: both sweeps of the pre-smoothing from z = 0 with the residual
// and its restriction, or the coarse correction and both sweeps of the post-smoothing. Over tiles
// held in registers: a block takes a region of 64 columns by R = MG_WARPS RPW rows, a lane two
// neighbouring columns of its warp's RPW rows (z, r, diag, 1/diag or omega/diag, east, south of
// each cell). A pass's horizontal neighbours come from the next lane by a shuffle, its vertical ones
// from the lane's own rows, or for a warp's first and last row from the neighbouring warp's through
// shared memory (one barrier a pass). The region's rim computes without its outer neighbours; what
// that spoils moves in one ring a pass (the first pass from z = 0 spoils none), so the tile is the
// region less H rings: 4 for the Gauss-Seidel sweeps (4 colour passes, or 3 and the residual), 2
// for the Jacobi ones. Each cell's terms are mg_apply_at's in its order (which takes the west term
// before the east one in the last column of a wrapping level), so the values are the separate
// launches'. Cells outside the raster hold zeros, couplings included; x wraps in the loads.
//   RB, PRE    colours 0, 1, 0, 1;  !PRE  colours 1, 0, 1, 0 (colour: (i + j) % 2, so a level of two
//              colours: no wrap, or an even width)
//   Jacobi     z = wd r and one sweep; !PRE two sweeps
// !PRE reads z around its tile, which neighbouring tiles finish at the same time: it writes another
// buffer (zout = L.t). Levels of fewer than 2^31 cells (32-bit offsets). VEC: an even width, so
// that a lane's two columns are one aligned word.
// Bound by HBM on the largest levels: 25 (PRE) and 29 bytes a cell in FP32. The earlier form kept
// the six arrays in shared memory in red-black order (12 reads an update, 360 thread instructions
// a cell): FP32 8192 x 4096 PRE 505 us, !PRE 482 with the L2 flushed; this 164 (0.78 of the measured
// copy rate) and 222; 2048 x 1024 45 and 44 to 20 and 26. For the Jacobi cycle it takes the place of
// three launches each way: a 2048 x 656 cycle of 49 launches becomes 11.
// Regions: 64 rows in FP32 on levels of many tiles (the rim is 1.3 times the tile), else 32.
constexpr int MG_WARPS = 16;
template <class TM>
struct Pair2 {
  TM v[2];
};
template <class TM, bool VEC>
__device__ __forceinline__ Pair2<TM> mg_load2(const TM* __restrict__ a, int row, int c0, int c1, bool ok0, bool ok1) {
  Pair2<TM> p;
  if constexpr (VEC) {
    using V = typename std::conditional<sizeof(TM) == 4, float2, double2>::type;
    V t;
    t.x = t.y = (TM)0;
    if (ok0) t = *reinterpret_cast<const V*>(a + (row + c0));
    p.v[0] = t.x;
    p.v[1] = t.y;
  } else {
    p.v[0] = ok0 ? a[row + c0] : (TM)0;
    p.v[1] = ok1 ? a[row + c1] : (TM)0;
  }
  return p;
}

//
// DOT (the finest level's post-smoothing in an FP32 CG): r . z too, so that the two are not read again
// for it (62 us at 8192 x 4096).
template <class TM, bool RB, bool PRE, int RPW, bool VEC, bool DOT>
__global__ void __launch_bounds__(32 * MG_WARPS, sizeof(TM) == 4 ? 2 : 1)
    k_mg_tile(DLevel<TM> L, DLevel<TM> C, const TM* __restrict__ zc, TM* __restrict__ zout, double* partials, DScalars* S) {
  static_assert(!(PRE && DOT), "r . z of the cycle's result");
  constexpr int H = RB ? 4 : 2, R = MG_WARPS * RPW, TX = 64 - 2 * H, TY = R - 2 * H;
  static_assert(RPW % 2 == 0 && TX % 2 == 0 && TY % 2 == 0, "even rows: a cell's colour and its coarse cell are known per row");
  // the warps' first and last rows, two buffers by pass
  __shared__ Pair2<TM> edge[2][2][MG_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w = L.w, h = L.h;
  const int raw = (int)blockIdx.x * TX - H + 2 * lane, j0 = (int)blockIdx.y * TY - H + warp * RPW;
  int c0 = raw, c1 = raw + 1;
  bool ok0 = c0 >= 0 && c0 < w, ok1 = c1 >= 0 && c1 < w;
  if (L.wrap) {
    c0 %= w;
    c0 += c0 < 0 ? w : 0;
    c1 = c0 + 1 == w ? 0 : c0 + 1;
    ok0 = ok1 = true;
  }
  const bool seam0 = L.wrap && c0 == w - 1, seam1 = L.wrap && c1 == w - 1;
  Pair2<TM> z[RPW], r[RPW], dg[RPW], wd[RPW], es[RPW], so[RPW], so_up;
#pragma unroll
  for (int q = 0; q < RPW; ++q) {
    const int j = j0 + q;
    const bool in = j >= 0 && j < h;
    const int row = j * w;
    r[q] = mg_load2<TM, VEC>(L.r, row, c0, c1, in && ok0, in && ok1);
    wd[q] = mg_load2<TM, VEC>(L.wd, row, c0, c1, in && ok0, in && ok1);
    if (!PRE) z[q] = mg_load2<TM, VEC>(L.z, row, c0, c1, in && ok0, in && ok1);
    dg[q] = mg_load2<TM, VEC>(L.diag, row, c0, c1, in && ok0, in && ok1);
    es[q] = mg_load2<TM, VEC>(L.east, row, c0, c1, in && ok0, in && ok1);
    so[q] = mg_load2<TM, VEC>(L.south, row, c0, c1, in && ok0, in && ok1);
  }
  {
    const bool in = j0 > 0 && j0 <= h;
    so_up = mg_load2<TM, VEC>(L.south, (j0 - 1) * w, c0, c1, in && ok0, in && ok1);
  }
  if constexpr (PRE) {
#pragma unroll
    for (int q = 0; q < RPW; ++q)
#pragma unroll
      for (int c = 0; c < 2; ++c) z[q].v[c] = !RB || ((q + c) & 1) == 0 ? (RB ? mulr(r[q].v[c], wd[q].v[c]) : wd[q].v[c] * r[q].v[c]) : (TM)0;
  } else {
#pragma unroll
    for (int q = 0; q < RPW; q += 2) {
      const int j = j0 + q;
      const bool in = j >= 0 && j < h;
      const int cr = (j >> 1) * C.w;
      const TM a = in && ok0 ? zc[cr + (c0 >> 1)] : (TM)0;
      const TM b = VEC ? a : (in && ok1 ? zc[cr + (c1 >> 1)] : (TM)0);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (in && (u == 0 || j + 1 < h)) {
          z[q + u].v[0] += a;
          z[q + u].v[1] += b;
        }
      }
    }
  }
  TM ew[RPW];  // the west neighbour's east coupling of the even columns
#pragma unroll
  for (int q = 0; q < RPW; ++q) ew[q] = __shfl_up_sync(0xffffffffu, es[q].v[1], 1);
  int buf = 0;
  auto publish = [&](int b) {
    edge[b][0][warp][lane] = z[0];
    edge[b][1][warp][lane] = z[RPW - 1];
  };
  // A z at the lane's cell (q, c) from its row's and neighbours' values
  auto apply = [&](int q, int c, TM zk, TM ze, TM zw, TM zn, TM zs) {
    TM o = mulr(dg[q].v[c], zk);
    const TM a = mulr(es[q].v[c], ze), b = mulr(c ? es[q].v[0] : ew[q], zw);
    const bool seam = c ? seam1 : (!VEC && seam0);
    o -= seam ? b : a;
    o -= seam ? a : b;
    o -= mulr(so[q].v[c], zs);
    o -= mulr(q ? so[q ? q - 1 : 0].v[c] : so_up.v[c], zn);
    return o;
  };
  auto neighbours = [&](Pair2<TM>& up, Pair2<TM>& down) {
    up.v[0] = up.v[1] = down.v[0] = down.v[1] = (TM)0;
    if (warp > 0) up = edge[buf][1][warp - 1][lane];
    if (warp < MG_WARPS - 1) down = edge[buf][0][warp + 1][lane];
  };
  constexpr int PASSES = RB ? (PRE ? 3 : 4) : (PRE ? 1 : 2);
  publish(0);
  __syncthreads();
#pragma unroll
  for (int pass = 0; pass < PASSES; ++pass) {
    Pair2<TM> up, down;
    neighbours(up, down);
    if constexpr (RB) {
      const int k = 1 - (pass & 1);  // PRE: the first pass (colour 0) is done; both go 1, 0, 1(, 0)
#pragma unroll
      for (int q = 0; q < RPW; ++q) {
        const int c = (k + q) & 1;  // the row's column of colour k
        const TM zk = z[q].v[c], in = z[q].v[1 - c];
        const TM out = c ? __shfl_down_sync(0xffffffffu, in, 1) : __shfl_up_sync(0xffffffffu, in, 1);
        const TM zn = q ? z[q ? q - 1 : 0].v[c] : up.v[c], zs = q + 1 < RPW ? z[q + 1 < RPW ? q + 1 : q].v[c] : down.v[c];
        const TM o = apply(q, c, zk, c ? out : in, c ? in : out, zn, zs);
        z[q].v[c] = zk + mulr(r[q].v[c] - o, wd[q].v[c]);
      }
    } else {
      Pair2<TM> prev = up;  // the row above before this sweep
#pragma unroll
      for (int q = 0; q < RPW; ++q) {
        const Pair2<TM> old = z[q], next = q + 1 < RPW ? z[q + 1 < RPW ? q + 1 : q] : down;
        const TM zr = __shfl_down_sync(0xffffffffu, old.v[0], 1), zl = __shfl_up_sync(0xffffffffu, old.v[1], 1);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const TM az = apply(q, c, old.v[c], c ? zr : old.v[1], c ? old.v[0] : zl, prev.v[c], next.v[c]);
          z[q].v[c] = old.v[c] + wd[q].v[c] * (r[q].v[c] - az);
        }
        prev = old;
      }
    }
    if (PRE || pass + 1 < PASSES) {
      publish(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
  const bool lanes_in = lane >= H / 2 && lane < 32 - H / 2;
  if constexpr (PRE) {
    Pair2<TM> up, down;
    neighbours(up, down);
    TM acc = 0;
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const Pair2<TM> next = q + 1 < RPW ? z[q + 1 < RPW ? q + 1 : q] : down, prev = q ? z[q ? q - 1 : 0] : up;
      const TM zr = __shfl_down_sync(0xffffffffu, z[q].v[0], 1), zl = __shfl_up_sync(0xffffffffu, z[q].v[1], 1);
      if ((q & 1) == 0) acc = (TM)0;
      const TM a0 = r[q].v[0] - apply(q, 0, z[q].v[0], z[q].v[1], zl, prev.v[0], next.v[0]);
      const TM a1 = r[q].v[1] - apply(q, 1, z[q].v[1], zr, z[q].v[0], prev.v[1], next.v[1]);
      if (j0 + q < h) {
        acc += a0;
        if (VEC || raw + 1 < w) acc += a1;
      }
      if (q & 1) {
        const int j = j0 + q - 1, rr = warp * RPW + q - 1;
        if (lanes_in && raw < w && rr >= H && rr < R - H && j < h) C.r[(j >> 1) * C.w + (raw >> 1)] = acc;
      }
    }
  }
  Acc<1> acc;
  acc.v[0] = 0.0;
#pragma unroll
  for (int q = 0; q < RPW; ++q) {
    const int j = j0 + q, rr = warp * RPW + q, at = j * w + raw;
    if (!lanes_in || raw >= w || rr < H || rr >= R - H || j >= h) continue;
    if constexpr (VEC) {
      using V = typename std::conditional<sizeof(TM) == 4, float2, double2>::type;
      V t;
      t.x = z[q].v[0];
      t.y = z[q].v[1];
      *reinterpret_cast<V*>(zout + at) = t;
    } else {
      zout[at] = z[q].v[0];
      if (raw + 1 < w) zout[at + 1] = z[q].v[1];
    }
    if constexpr (DOT) {
      acc.v[0] += (double)r[q].v[0] * (double)z[q].v[0];
      if (VEC || raw + 1 < w) acc.v[0] += (double)r[q].v[1] * (double)z[q].v[1];
    }
  }
  if constexpr (DOT) {
    if (S->stop) return;
    const int kind[1] = {0};
    if (reduce_partials<1>(acc, kind, partials, &S->ticket[DSITE_RZ], gridDim.x * gridDim.y) && threadIdx.x == 0)
      d_finish_rz(S, acc.v[0]);
  }
}

// ---------------------------------------------------------------------------------------------
// LOD first guess (diffusion.rs:370-489): an implicit sweep along x per row (cyclic tridiagonal,
// Sherman-Morrison, :1050-1071) and then along y per column (Thomas, :1029-1046). One thread
// per row or column; scratch arrays of the raster's size.

__device__ void thomas_strided(int n, const double* lo, const double* di, const double* up, double* b, double* c, size_t stride,
                               size_t base) {
  // lo/di/up/b/c accessed at base + i * stride
  if (n == 0) return;
  double beta = di[base];
  b[base] /= beta;
  for (int i = 1; i < n; ++i) {
    size_t at = base + (size_t)i * stride, prev = at - stride;
    c[at] = up[prev] / beta;
    beta = di[at] - lo[at] * c[at];
    b[at] = (b[at] - lo[at] * b[prev]) / beta;
  }
  for (int i = n - 2; i >= 0; --i) {
    size_t at = base + (size_t)i * stride;
    double next = b[at + stride];
    b[at] -= c[at + stride] * next;
  }
}

__global__ void k_lod_rows(int w, int h, int wrap, double* __restrict__ hf, const double* __restrict__ kd, double dtdx2,
                           double* lo, double* di, double* up, double* xs, double* zs, double* cs) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= h) return;
  size_t c0 = (size_t)j * w;
  const double* krow = kd + c0;
  auto face = [&](int i) -> double {
    if (i + 1 < w) return 0.5 * (krow[i] + krow[i + 1]) * dtdx2;
    if (wrap && w > 1) return 0.5 * (krow[w - 1] + krow[0]) * dtdx2;
    return 0.0;
  };
  for (int i = 0; i < w; ++i) {
    double west = i == 0 ? face(w - 1) : face(i - 1);
    double east = face(i);
    lo[c0 + i] = -west;
    up[c0 + i] = -east;
    di[c0 + i] = 1.0 + west + east;
  }
  if (wrap && w > 2) {
    // cyclic: corners alpha = up[w-1] (row w-1, column 0), beta = lo[0] (row 0, column w-1)
    double alpha = up[c0 + w - 1], beta = lo[c0];
    double gamma = -di[c0];
    di[c0] = di[c0] - gamma;
    di[c0 + w - 1] = di[c0 + w - 1] - alpha * beta / gamma;
    lo[c0] = 0.0;
    up[c0 + w - 1] = 0.0;
    for (int i = 0; i < w; ++i) {
      xs[c0 + i] = hf[c0 + i];
      zs[c0 + i] = 0.0;
    }
    zs[c0] = gamma;
    zs[c0 + w - 1] = alpha;
    thomas_strided(w, lo, di, up, xs, cs, 1, c0);
    thomas_strided(w, lo, di, up, zs, cs, 1, c0);
    double fact = (xs[c0] + beta * xs[c0 + w - 1] / gamma) / (1.0 + zs[c0] + beta * zs[c0 + w - 1] / gamma);
    for (int i = 0; i < w; ++i) hf[c0 + i] = xs[c0 + i] - fact * zs[c0 + i];
  } else {
    if (w == 2 && wrap) {
      double f = face(0) + face(1);
      lo[c0 + 1] = -f;
      up[c0] = -f;
      di[c0] = 1.0 + f;
      di[c0 + 1] = 1.0 + f;
    }
    lo[c0] = 0.0;
    up[c0 + w - 1] = 0.0;
    if (w == 1) di[c0] = 1.0;
    thomas_strided(w, lo, di, up, hf, cs, 1, c0);
  }
}

// The LOD passes as partitioned tridiagonal solves: L independent lines of n unknowns, rows as they
// lie (ROWS: the periodic rows, element (l, i) at l n + i) or columns (element (l, i) at i L + l).
// A block takes G lines (columns: neighbouring ones, a row's segment of G words) over a segment of
// 16 Pb unknowns, a thread 16 of them in registers:
//   1. Thomas's elimination of the thread's chunk (diffusion.rs:1029-1046), with the chunk's first and
//      last values as A = pA + qA y_left + rA y_right, B = pB + qB y_left + rB y_right, y_left and
//      y_right the unknowns just outside it;
//   2. neighbouring chunks merged pairwise up a tree in shared memory to the segment's own relation,
//      and the outside values handed down it again;
//   3. the chunk's solution from its outside values.
// So kd and the right-hand side are read once and the solution written once (24 bytes a cell). Bound
// by latency (16 dependent reciprocals, two passes over log2(Pb) tree levels) below about a wave of
// blocks, then by HBM. As separate passes over scratch arrays, with the rows on transposed copies, the
// two directions took 2.6 ms at 8192 x 4096 and 330 us at 2048 x 1024; this 1.1 ms and 65 us.
// The coefficients are the LOD's (diffusion.rs:370-489), formed from kd: faces 0.5 (k_i + k_(i+1))
// dt / dx^2 and diagonal (1 + west) + east. ROWS: Sherman-Morrison (diffusion.rs:1048-1071): the
// corners folded into the first and last diagonal, solved for b and u = (gamma, 0, .., 0, alpha), then
// x - fact z; u's response rides along as a second p, and the last step solves for b - fact u.
// Lines of more than a segment: STEP 1 writes each segment's relation, k_lod_reduce solves those a
// line, STEP 2 solves the segments between their outside values (kd and b read twice). STEP 0: one
// segment a line.
constexpr int LOD_CH = 16, LOD_THREADS = 512;
template <bool ROWS>
struct LodLine {
  const double* kd;
  int L, n, l;
  double dtdx2;
  __device__ double K(int i) const { return ROWS ? kd[(size_t)l * n + i] : kd[(size_t)i * L + l]; }
  // the face between positions i and i + 1 (across the seam for the rows' last one)
  __device__ double face(int i) const {
    if (i + 1 < n) return 0.5 * (K(i) + K(i + 1)) * dtdx2;
    return ROWS ? 0.5 * (K(n - 1) + K(0)) * dtdx2 : 0.0;
  }
};
// shared memory: 8 values a chunk's relation, 4 its outside values, and for the rows their kd and
// right-hand side, spaced by one word after every 16 so that the threads' chunks fall in distinct banks
__host__ __device__ constexpr size_t lod_smem(bool rows) {
  return (size_t)LOD_THREADS * (12 + (rows ? 2 * (LOD_CH + 1) : 0)) * sizeof(double);
}
template <bool ROWS, int STEP>
__global__ void __launch_bounds__(LOD_THREADS, 1) k_lod_lines(int L, int n, int Pb, int G, double dtdx2, const double* kd,
                                                              const double* b, double* x, double* edge, const double* fact) {
  extern __shared__ __align__(16) unsigned char lod_raw[];
  double* const rel = reinterpret_cast<double*>(lod_raw);  // [8][threads]: pA0, pA1, qA, rA, pB0, pB1, qB, rB
  double* const out = rel + 8 * LOD_THREADS;               // [4][threads]: y_left for b, for u; y_right for b, for u
  double* const sk = out + 4 * LOD_THREADS;                // ROWS: kd, then b, of the block's lines
  double* const sb = sk + LOD_THREADS * (LOD_CH + 1);
  __shared__ double s_fact[LOD_THREADS];
  const int tid = threadIdx.x, nt = Pb * G;
  const int c = ROWS ? tid % Pb : tid / G, g = ROWS ? tid / Pb : tid % G;
  const int l = blockIdx.x * G + g, s0 = blockIdx.y * Pb * LOD_CH, s = s0 + c * LOD_CH;
  const bool on = tid < nt && l < L;
  const int len = on ? min(max(n - s, 0), LOD_CH) : 0;
  const int chunks = (min(n - s0, Pb * LOD_CH) + LOD_CH - 1) / LOD_CH;  // of this segment
  const LodLine<ROWS> ln{kd, L, n, l, dtdx2};
  double kv[LOD_CH + 2], p[LOD_CH], m[LOD_CH], cc[LOD_CH];  // kv: columns only, kd of s - 1 .. s + LOD_CH
  double k_before = 0.0, k_after = 0.0, k_first = 0.0, k_last = 0.0;
  if constexpr (ROWS) {
    const int width = min(n - s0, Pb * LOD_CH), lines = min(G, L - (int)blockIdx.x * G);
    for (int e = tid; e < lines * width; e += blockDim.x) {
      const int ge = e / width, i = e - ge * width;
      const size_t src = (size_t)(blockIdx.x * G + ge) * n + s0 + i;
      const int dst = ge * Pb * (LOD_CH + 1) + i + i / LOD_CH;
      __pipeline_memcpy_async(sk + dst, kd + src, 8);
      __pipeline_memcpy_async(sb + dst, b + src, 8);
    }
    __pipeline_commit();
    if (len > 0) {
      if (s > 0) k_before = ln.K(s - 1);
      if (s + len < n) k_after = ln.K(s + len);
      k_first = ln.K(0);
      k_last = ln.K(n - 1);
    }
    __pipeline_wait_prior(0);
    __syncthreads();
  } else {
#pragma unroll
    for (int t = 0; t < LOD_CH + 2; ++t) {
      const int i = s + t - 1;
      kv[t] = len > 0 && i >= 0 && i < n ? ln.K(i) : 0.0;
    }
#pragma unroll
    for (int t = 0; t < LOD_CH; ++t) p[t] = t < len ? b[(size_t)(s + t) * L + l] : 0.0;
  }
  double* const mk = sk + (g * Pb + c) * (LOD_CH + 1);
  double* const mb = sb + (g * Pb + c) * (LOD_CH + 1);

  // rows: the folded corners (k_lod_rows' alpha = up[n-1], beta = lo[0], gamma = -di[0])
  double fw = 0.0, alpha = 0.0, gamma = -1.0;
  if (ROWS && len > 0) {
    fw = 0.5 * (k_last + k_first) * dtdx2;
    alpha = -fw;
    if (s == 0) gamma = -(1.0 + fw + 0.5 * (k_first + (len > 1 ? mk[1] : k_after)) * dtdx2);
    else if (s + len == n) gamma = -(1.0 + fw + ln.face(0));
  }
  double lo0 = 0.0, ib0 = 0.0, ibl = 0.0;
  // kd of the chunk's unknowns t = -1 .. len
  auto K = [&](int t) {
    if constexpr (ROWS)
      return t < 0 ? k_before : t < len ? mk[t] : k_after;
    else
      return kv[t + 1];
  };
  {
    double west = s == 0 ? (ROWS ? fw : 0.0) : 0.5 * (K(-1) + K(0)) * dtdx2, last_c = 0.0;
    double pv = 0.0, ev = 0.0, pA0 = 0.0, pA1 = 0.0, eA = 0.0, rA = 1.0;
#pragma unroll
    for (int t = 0; t < LOD_CH; ++t) {
      m[t] = cc[t] = 0.0;
      if (t < len) {
        const int i = s + t;
        const bool end = i == n - 1;
        const double east = end ? (ROWS ? fw : 0.0) : 0.5 * (K(t) + K(t + 1)) * dtdx2;
        double di = 1.0 + west + east;
        if (ROWS && i == 0) di = di - gamma;
        if (ROWS && end) di = di - alpha * alpha / gamma;  // beta = alpha
        const double lo = i == 0 ? 0.0 : -west, up = end ? 0.0 : -east;
        const double ib = recip(t == 0 ? di : di - lo * cc[t > 0 ? t - 1 : 0]);
        m[t] = lo * ib;
        cc[t] = up * ib;
        const double b0 = (ROWS ? mb[t] : p[t]) * ib;
        if (t == 0) {
          lo0 = lo;
          ib0 = ib;
          pv = b0;
          ev = ib;  // the response to a unit right-hand side at the chunk's first unknown
        } else {
          pv = b0 - m[t] * pv;
          ev = -m[t] * ev;
        }
        p[t] = pv;
        // y_first = pA + eA u + rA y_next, one unknown further each step
        pA0 += rA * pv;
        eA += rA * ev;
        if (ROWS && end) {
          pA1 = rA * (alpha * ib);
          ibl = ib;
        }
        rA *= -cc[t];
        last_c = cc[t];
        west = east;
      }
    }
    if (on) {
      const double u0 = ROWS && s == 0 ? gamma : 0.0;
      rel[0 * LOD_THREADS + tid] = pA0;
      rel[1 * LOD_THREADS + tid] = u0 * eA + pA1;
      rel[2 * LOD_THREADS + tid] = -lo0 * eA;
      rel[3 * LOD_THREADS + tid] = rA;
      rel[4 * LOD_THREADS + tid] = pv;
      rel[5 * LOD_THREADS + tid] = u0 * ev + (ROWS && len > 0 && s + len == n ? alpha * ibl : 0.0);
      rel[6 * LOD_THREADS + tid] = -lo0 * ev;
      rel[7 * LOD_THREADS + tid] = -last_c;
    }
  }
  __syncthreads();
  // up the tree: the relations of chunks [c, c + 2^k) and [c + 2^k, c + 2^(k+1)) merge into c's slot; the
  // values they meet at, first of the right and last of the left part, as relations to the merged
  // chunk's outside, take the right part's slot
  const int step = ROWS ? 1 : G;  // a chunk's neighbour's slot
  auto R = [&](int k, int t) -> double& { return rel[k * LOD_THREADS + t]; };
  int levels = 0;
  for (; (1 << levels) < chunks; ++levels) {
    const int d = 1 << levels, t2 = tid + d * step;
    if (on && (c & (2 * d - 1)) == 0 && c + d < chunks) {
      const double qA2 = R(2, t2), rB1 = R(7, tid), qB1 = R(6, tid), rA1 = R(3, tid), qB2 = R(6, t2);
      const double D = recip(1.0 - qA2 * rB1);
      const double a0 = D * (R(0, t2) + qA2 * R(4, tid)), aq = D * (qA2 * qB1), ar = D * R(3, t2);
      const double b0 = R(4, tid) + rB1 * a0, bq = qB1 + rB1 * aq, br = rB1 * ar;
      R(0, tid) += rA1 * a0;
      R(2, tid) += rA1 * aq;
      R(3, tid) = rA1 * ar;
      const double pB = R(4, t2) + qB2 * b0, rB = R(7, t2) + qB2 * br;
      if (ROWS) {
        const double a1 = D * (R(1, t2) + qA2 * R(5, tid)), b1 = R(5, tid) + rB1 * a1;
        R(1, tid) += rA1 * a1;
        R(5, tid) = R(5, t2) + qB2 * b1;
        R(1, t2) = a1;
        R(5, t2) = b1;
      }
      R(4, tid) = pB;
      R(6, tid) = qB2 * bq;
      R(7, tid) = rB;
      R(0, t2) = a0;
      R(2, t2) = aq;
      R(3, t2) = ar;
      R(4, t2) = b0;
      R(6, t2) = bq;
      R(7, t2) = br;
    }
    __syncthreads();
  }
  const size_t seg = (size_t)blockIdx.y * L + l;
  if constexpr (STEP == 1) {
    if (on && c == 0)
      for (int k = 0; k < 8; ++k) edge[seg * 8 + k] = R(k, tid);
    return;
  }
  if (on && c == 0) {
    double y[4] = {0.0, 0.0, 0.0, 0.0}, f = 0.0;
    if constexpr (STEP == 2) {
      if (blockIdx.y > 0) {
        const double* em = edge + (seg - L) * 8;
        y[0] = em[4];
        if (ROWS) y[1] = em[5];
      }
      if (blockIdx.y + 1 < gridDim.y) {
        const double* ep = edge + (seg + L) * 8;
        y[2] = ep[0];
        if (ROWS) y[3] = ep[1];
      }
      if (ROWS) f = fact[l];
    } else if (ROWS) {
      // the line's own first and last values: the root's, with nothing outside
      f = (R(0, tid) + alpha * R(4, tid) / gamma) / (1.0 + R(1, tid) + alpha * R(5, tid) / gamma);
    }
    for (int k = 0; k < 4; ++k) out[k * LOD_THREADS + tid] = y[k];
    if (ROWS) s_fact[g] = f;
  }
  // down the tree: the outside values of each half from the whole's
  for (int k = levels - 1; k >= 0; --k) {
    __syncthreads();
    const int d = 1 << k, t2 = tid + d * step;
    if (on && (c & (2 * d - 1)) == 0 && c + d < chunks) {
      const double L0 = out[tid], R0 = out[2 * LOD_THREADS + tid];
      out[t2] = R(4, t2) + R(6, t2) * L0 + R(7, t2) * R0;
      out[2 * LOD_THREADS + t2] = R0;
      out[2 * LOD_THREADS + tid] = R(0, t2) + R(2, t2) * L0 + R(3, t2) * R0;
      if (ROWS) {
        const double L1 = out[LOD_THREADS + tid], R1 = out[3 * LOD_THREADS + tid];
        out[LOD_THREADS + t2] = R(5, t2) + R(6, t2) * L1 + R(7, t2) * R1;
        out[3 * LOD_THREADS + t2] = R1;
        out[3 * LOD_THREADS + tid] = R(1, t2) + R(2, t2) * L1 + R(3, t2) * R1;
      }
    }
  }
  __syncthreads();
  if (len > 0) {
    const double f = ROWS ? s_fact[g] : 0.0;
    const double left = out[tid] - (ROWS ? f * out[LOD_THREADS + tid] : 0.0);
    const double right = out[2 * LOD_THREADS + tid] - (ROWS ? f * out[3 * LOD_THREADS + tid] : 0.0);
    // b - fact u, with the outside values on the right-hand side
    double ev = (-lo0 * left - (ROWS && s == 0 ? f * gamma : 0.0)) * ib0;
#pragma unroll
    for (int t = 0; t < LOD_CH; ++t) {
      if (t > 0) ev = -m[t] * ev;
      p[t] += ev;
      if (ROWS && t < len && s + t == n - 1) p[t] -= f * (alpha * ibl);
    }
    double y = right;
#pragma unroll
    for (int t = LOD_CH - 1; t >= 0; --t) {
      if (t < len) {
        y = p[t] - cc[t] * y;
        if (ROWS)
          mb[t] = y;
        else
          x[(size_t)(s + t) * L + l] = y;
      }
    }
  }
  if constexpr (ROWS) {
    __syncthreads();
    const int width = min(n - s0, Pb * LOD_CH), lines = min(G, L - (int)blockIdx.x * G);
    for (int e = tid; e < lines * width; e += blockDim.x) {
      const int ge = e / width, i = e - ge * width;
      x[(size_t)(blockIdx.x * G + ge) * n + s0 + i] = sb[ge * Pb * (LOD_CH + 1) + i + i / LOD_CH];
    }
  }
}

// One thread a line: the segments' first (A_k) and last (B_k) values from A_k = pA + qA B_(k-1) +
// rA A_(k+1), B_k = pB + qB B_(k-1) + rB A_(k+1): forward, B_(k-1) = g + h A_k; back from A_P = 0.
// Written over the edge record's p entries (A_k into [0], [1], B_k into [4], [5]); ROWS: fact of
// the line into fact[l].
template <bool ROWS>
__global__ void __launch_bounds__(128) k_lod_reduce(int L, int n, int P, double dtdx2, const double* __restrict__ kd,
                                                    double* __restrict__ edge, double* __restrict__ al,
                                                    double* __restrict__ fact) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= L) return;
  constexpr int NR = ROWS ? 2 : 1;
  double A0[NR], Bl[NR];
  for (int rhs = 0; rhs < NR; ++rhs) {
    double g = 0.0, hh = 0.0;
    for (int k = 0; k < P; ++k) {
      const double* ed = edge + ((size_t)k * L + l) * 8;
      const double pA = ed[rhs], qA = ed[2], rA = ed[3], pB = ed[4 + rhs], qB = ed[6], rB = ed[7];
      const double d = 1.0 - qA * hh;
      const double a = (pA + qA * g) / d, be = rA / d;
      // scratch for the way back: alpha, beta, g, h of chunk k
      double* sk = al + ((size_t)k * L + l) * 4;
      sk[0] = a;
      sk[1] = be;
      g = pB + qB * g + qB * hh * a;
      hh = qB * hh * be + rB;
      sk[2] = g;
      sk[3] = hh;
    }
    double An = 0.0;
    for (int k = P - 1; k >= 0; --k) {
      const double* sk = al + ((size_t)k * L + l) * 4;
      const double A = sk[0] + sk[1] * An, B = sk[2] + sk[3] * An;
      double* ed = edge + ((size_t)k * L + l) * 8;
      ed[rhs] = A;
      ed[4 + rhs] = B;
      if (k == P - 1) Bl[rhs] = B;
      An = A;
    }
    A0[rhs] = An;
  }
  if (ROWS) {
    const LodLine<true> ln{kd, L, n, l, dtdx2};
    const double fw = ln.face(n - 1);
    const double beta = -fw, gamma = -(1.0 + fw + ln.face(0));
    fact[l] = (A0[0] + beta * Bl[0] / gamma) / (1.0 + A0[1] + beta * Bl[1] / gamma);
  }
}

// ---------------------------------------------------------------------------------------------
// Small control kernels.

__global__ void k_d_arm(DScalars* S, unsigned long long handle, unsigned long long handle_if) {
  S->cond = handle;
  S->cond_if = handle_if;
  S->body_runs = 0;
  cudaGraphSetConditional((cudaGraphConditionalHandle)handle, S->stop == 0 ? 1u : 0u);
}
// dt_diff_profile_kernels: a solve's state record ready for one more operator launch
__global__ void k_d_profile_state(DScalars* S) {
  S->stop = 0;
  S->cond = 0ull;
}
__global__ void k_d_disarm(DScalars* S) {
  S->cond = 0ull;
  S->cond_if = 0ull;
}

struct DProblem {
  double tol;
  int max_it, rule, n;
  int reliable;  // the FP32 lane of DT_DIFF_MIXED_RELIABLE (its other fields from k_d_rel_init)
};
__global__ void k_d_begin(DScalars* S, DProblem p, int bb_from_dot) {
  S->tol = p.tol;
  S->max_it = p.max_it;
  S->rule = p.rule;
  S->n = p.n;
  if (bb_from_dot) S->bb = S->dot_out;
  S->it = 0;
  S->stop = 0;
  S->started = 0;
  S->body_runs = 0;
  S->cond = 0ull;
  S->reliable = p.reliable;
  S->gate_it = -1;
  if (!isfinite(S->rr) || !isfinite(S->bb))
    S->stop = DSTOP_NONFINITE;
  else if (!(S->rr > 0.0) || d_converged(S, S->rr))
    S->stop = DSTOP_CONVERGED;
}

template <class T>
__global__ void __launch_bounds__(256) k_d_dot(size_t n, const T* __restrict__ a, const T* __restrict__ b, double* partials,
                                               DScalars* S) {
  Acc<1> acc;
  acc.v[0] = 0.0;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    acc.v[0] += (double)a[k] * (double)b[k];
  const int kind[1] = {0};
  if (reduce_partials<1>(acc, kind, partials, &S->ticket[DSITE_DOT], gridDim.x) && threadIdx.x == 0) S->dot_out = acc.v[0];
}

// x += (lost / weight)(diag - 1) when weight > 0 and lost != 0 (multigrid.rs:755-761)
__global__ void k_d_massfix(size_t n, double* __restrict__ x, const double* __restrict__ diag, const DScalars* S) {
  double lost = S->lost, weight = S->weight;
  if (!(weight > 0.0 && lost != 0.0)) return;
  double k = lost / weight;
  for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) x[c] += k * (diag[c] - 1.0);
}

__global__ void k_d_scale_down(size_t n, const double* __restrict__ r, float* __restrict__ r32, float* __restrict__ x32,
                               const DScalars* S64, double* scale) {
  double s = S64->rr > 0 ? sqrt((double)n / S64->rr) : 1.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *scale = s;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    r32[k] = (float)(r[k] * s);
    x32[k] = 0.0f;
  }
}
__global__ void k_d_accumulate(size_t n, double* __restrict__ x, const float* __restrict__ x32, const double* scale) {
  double inv = 1.0 / *scale;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) x[k] += (double)x32[k] * inv;
}
__global__ void k_d_rr_is_bb(DScalars* S) { S->rr = S->bb; }

// Reliable updates (the FP32 lane holds r32 = s r64 and its correction x32 = s e, s fixed from the
// first residual's RMS). In an iteration that replaces the residual (gate_it == it):
//   k_d_rel_accumulate                x64 += x32 / s; x32 = 0
//   k_d_apply<.., DA_RESID_GATED>     r64 = b - A x64, ||r64||^2 -> rr_true
//   k_d_rel_reset                     r32 = s r64; rr, maxrr from rr_true;
//                                     stop when rr_true meets the tolerance
__global__ void k_d_rel_accumulate(size_t n, double* __restrict__ x, float* __restrict__ x32, const double* scale,
                                   const DScalars* S) {
  if (S->stop || S->gate_it != S->it) return;
  double inv = 1.0 / *scale;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    x[k] += (double)x32[k] * inv;
    x32[k] = 0.0f;
  }
}
__global__ void k_d_rel_reset(size_t n, const double* __restrict__ r, float* __restrict__ r32, const double* scale, DScalars* S) {
  if (S->stop || S->gate_it != S->it) return;
  double sc = *scale;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    r32[k] = (float)(r[k] * sc);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    double rr = S->rr_true * sc * sc;
    S->rr = rr;
    S->maxrr = rr;
    S->replacements += 1;
    if (!isfinite(S->rr_true)) {
      S->stop = DSTOP_NONFINITE;
    } else if (S->rr_true <= S->tol * S->tol * S->bb_true) {
      S->stop = DSTOP_CONVERGED;
    }
    if (S->stop) dset_cond(S, 0);
  }
}
// The FP32 lane's problem for reliable updates, from the FP64 lane's (bb, rr of r = b - A x) and
// the scale s of r32 = s r: the tolerance on the relative residual, or with `rms` on the RMS
// residual (||r||^2 <= tol^2 n).
__global__ void k_d_rel_init(DScalars* F, const DScalars* S64, const double* scale, double delta, int rms) {
  double s2 = (*scale) * (*scale);
  double bref = rms ? (double)S64->n : S64->bb;
  F->bb = bref * s2;
  F->bb_true = bref;
  F->rr = S64->rr * s2;
  F->maxrr = F->rr;
  F->delta2 = delta * delta;
  F->replacements = 0;
  F->cond_if = 0ull;
}
__global__ void k_convert_dr(size_t n, const double* __restrict__ a, float* __restrict__ b) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) b[k] = (float)a[k];
}

}  // namespace dt

// =============================================================================================
// Host side.

namespace dt {

static const float OMEGA = 0.8f;    // multigrid.rs:45
static const int NU = 2;            // multigrid.rs:48
static const float SCALE = 0.5f;    // multigrid.rs:52
static const int COARSEST = 64;     // multigrid.rs:54
static const int COARSE_SWEEPS = 16;  // multigrid.rs:56
static const int COARSEST_GS = 128;   // the Gauss-Seidel cycle's coarsest level: 16 x 8 cells
static const int COARSE_SWEEPS_GS = 8;

template <class TM>
struct Hier {
  std::vector<DLevel<TM>> lv;
  bool built = false;
};

// CG lanes: 0 FP64 CG + FP32 cycle, 1 FP64 CG + FP64 cycle, 2 FP32 CG + FP32 cycle (mixed inner)
struct DGraph {
  cudaGraph_t g = nullptr;
  cudaGraphExec_t exec = nullptr;
  long long body_kernels = 0;
};

}  // namespace dt

struct dt_diff {
  int w = 0, h = 0, wrap = 0;
  double dx = 0;
  size_t n = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int sms = 148;
  std::vector<void*> allocs;
  size_t nalloc = 0;  // device allocations made (the DT_FAIL_ALLOC_AT test hook counts them)
  double *kd = nullptr, *b = nullptr, *x = nullptr, *r = nullptr, *p = nullptr, *ap = nullptr;
  double *east = nullptr, *south = nullptr, *diag = nullptr;
  float *east32 = nullptr, *south32 = nullptr, *diag32 = nullptr;
  float *x32 = nullptr, *r32 = nullptr, *p32 = nullptr, *ap32 = nullptr;
  double* lod[7] = {};  // the LOD first guess's scratch (lod[6]: its segments' relations)
  double* partials = nullptr;
  double* scale = nullptr;
  dt::DScalars *S64 = nullptr, *S32 = nullptr;
  dt::Hier<float> hf[2];
  dt::Hier<double> hd[2];
  dt::DGraph graph[4][2];  // [lane: 0 split, 1 FP64, 2 FP32 inner, 3 FP32 reliable][cycle]
  // the cycles' fused kernels (k_mg_tile, k_mg_coarse); DT_MG_FUSED=0 at
  // create keeps one launch per sweep or colour pass (the same values)
  bool mg_fused = true;
  // k_mg_tile's 64-row regions on FP32 levels of many tiles; DT_MG_BIG_TILES=0 at create keeps
  // 32-row ones everywhere (the same values)
  bool mg_big_tiles = true;
};

namespace dt {

template <class T>
static dt_status ddalloc(dt_diff* s, T** p, size_t count) {
  void* q = nullptr;
  if (alloc_fault(s->nalloc)) {
    set_error("cudaMalloc of %zu bytes failed: out of memory (DT_FAIL_ALLOC_AT)", count * sizeof(T));
    return DT_OOM;
  }
  cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
  if (e != cudaSuccess) {
    set_error("cudaMalloc of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? DT_OOM : DT_DEVICE_ERROR;
  }
  s->allocs.push_back(q);
  *p = reinterpret_cast<T*>(q);
  return DT_OK;
}

static unsigned int dgrid(const dt_diff* s, size_t n) {
  return std::max(1u, std::min<unsigned int>(ceil_div(n, 256), (unsigned)s->sms * 8));
}

static void finest_arrays(dt_diff* s, DLevel<float>& L) {
  L.east = s->east32;
  L.south = s->south32;
  L.diag = s->diag32;
  L.r = s->r32;
  L.mass = nullptr;
}
static void finest_arrays(dt_diff* s, DLevel<double>& L) {
  L.east = s->east;
  L.south = s->south;
  L.diag = s->diag;
  L.r = s->r;
  L.mass = nullptr;
}

// The level shapes of the hierarchy (multigrid.rs:117-123): halve (rounding up) until the level
// has at most `coarsest` cells or stops shrinking; x wraps on a level while it is wider than 1.
template <class TM>
static dt_status build_levels(dt_diff* s, Hier<TM>& H, int coarsest) {
  if (H.built) return DT_OK;
  int w = s->w, h = s->h, wrap = s->wrap && s->w > 1;
  for (;;) {
    DLevel<TM> L;
    L.w = w;
    L.h = h;
    L.wrap = wrap;
    size_t n = (size_t)w * h;
    for (TM** q : {&L.wd, &L.z, &L.t}) DT_TRY(ddalloc(s, q, n));
    if (H.lv.empty()) {
      // the finest level: the operator's coefficients and the CG's residual (FP64 CG around an FP32
      // cycle leaves that residual's FP32 copy there), every mass 1
      finest_arrays(s, L);
    } else {
      for (TM** q : {&L.east, &L.south, &L.diag, &L.mass, &L.r}) DT_TRY(ddalloc(s, q, n));
    }
    H.lv.push_back(L);
    int wc = (w + 1) / 2, hc = (h + 1) / 2;
    if ((long)w * h <= coarsest || (wc == w && hc == h)) break;
    wrap = wrap && wc > 1;
    w = wc;
    h = hc;
  }
  H.built = true;
  return DT_OK;
}

// Level coefficients for the current operator: the finest are the operator's, the rest by
// aggregation.
// wd: omega / diag for the damped-Jacobi cycle, 1 / diag for the Gauss-Seidel one.
template <class TM>
static void fill_levels(dt_diff* s, Hier<TM>& H, int kind, cudaStream_t st) {
  DLevel<TM>& f = H.lv[0];
  const TM omega = kind == DT_CYCLE_JACOBI ? (TM)OMEGA : (TM)1;
  k_mg_finest<TM><<<dgrid(s, s->n), 256, 0, st>>>(s->n, f.diag, omega, f.wd);
  count_launch();
  for (size_t l = 1; l < H.lv.size(); ++l) {
    size_t nc = (size_t)H.lv[l].w * H.lv[l].h;
    k_mg_coarsen<TM><<<dgrid(s, nc), 256, 0, st>>>(H.lv[l - 1], H.lv[l], (TM)SCALE);
    k_mg_diag<TM><<<dgrid(s, nc), 256, 0, st>>>(H.lv[l], omega);
    count_launch();
    count_launch();
  }
}

// An FP32 CG's r . z asked of its cycle: `done` once the finest level's post-smoothing forms it.
struct RzArg {
  DScalars* S;
  bool done;
};
// A level's smoothing by k_mg_tile (PRE: from z = 0, the restriction into C.r; else with the coarse
// correction zc).
template <class TM, bool RB, bool PRE, int RPW, bool DOT>
static void launch_tile_rows(dt_diff* s, const DLevel<TM>& L, const DLevel<TM>& C, const TM* zc, TM* zout, DScalars* S,
                             cudaStream_t st) {
  constexpr int H = RB ? 4 : 2;
  const dim3 tg(ceil_div(L.w, 64 - 2 * H), ceil_div(L.h, MG_WARPS * RPW - 2 * H));
  if (L.w % 2 == 0)
    k_mg_tile<TM, RB, PRE, RPW, true, DOT><<<tg, 32 * MG_WARPS, 0, st>>>(L, C, zc, zout, s->partials, S);
  else
    k_mg_tile<TM, RB, PRE, RPW, false, DOT><<<tg, 32 * MG_WARPS, 0, st>>>(L, C, zc, zout, s->partials, S);
}
template <class TM, bool RB, bool PRE, bool DOT>
static void launch_tile_dot(dt_diff* s, const DLevel<TM>& L, const DLevel<TM>& C, const TM* zc, TM* zout, DScalars* S,
                            cudaStream_t st) {
  // 64-row regions on FP32 levels where those alone make at least four tiles an SM (FP64 rows of
  // four would not fit the registers)
  if constexpr (sizeof(TM) == 4) {
    constexpr int H = RB ? 4 : 2;
    if (s->mg_big_tiles && (size_t)ceil_div(L.w, 64 - 2 * H) * ceil_div(L.h, 64 - 2 * H) >= (size_t)4 * s->sms) {
      launch_tile_rows<TM, RB, PRE, 4, DOT>(s, L, C, zc, zout, S, st);
      return;
    }
  }
  launch_tile_rows<TM, RB, PRE, 2, DOT>(s, L, C, zc, zout, S, st);
}
template <class TM, bool RB, bool PRE>
static void launch_tile(dt_diff* s, const DLevel<TM>& L, const DLevel<TM>& C, const TM* zc, TM* zout, cudaStream_t st,
                        RzArg* rz = nullptr) {
  count_launch();
  if constexpr (!PRE && sizeof(TM) == 4) {
    if (rz) {
      launch_tile_dot<TM, RB, PRE, true>(s, L, C, zc, zout, rz->S, st);
      rz->done = true;
      return;
    }
  }
  launch_tile_dot<TM, RB, PRE, false>(s, L, C, zc, zout, nullptr, st);
}
// k_mg_tile's 32-bit offsets, and its rows of tiles (24 cells at the least) on the grid's y extent, which
// ends at 65535; taller levels take the launches a sweep
template <class TM>
static bool tile_fits(const DLevel<TM>& L) {
  return (size_t)L.w * L.h < ((size_t)1 << 31) && ceil_div(L.h, 24) <= 65535;
}

// One V-cycle from z = 0 on level l with r set; returns the buffer holding the level's z. With `rz` on
// the finest level, r . z as well where its post-smoothing forms it (rz->done).
template <class TM>
static TM* vcycle(dt_diff* s, Hier<TM>& H, size_t l, int kind, cudaStream_t st, RzArg* rz = nullptr) {
  DLevel<TM>& L = H.lv[l];
  size_t n = (size_t)L.w * L.h;
  unsigned int g = dgrid(s, n);
  bool coarsest = l + 1 == H.lv.size();
  if (coarsest) {
    if (kind == DT_CYCLE_JACOBI)
      k_mg_coarsest<TM, 0><<<1, 256, 0, st>>>(L, L.z, COARSE_SWEEPS);
    else
      k_mg_coarsest<TM, 1><<<1, 256, 0, st>>>(L, L.z, COARSE_SWEEPS_GS);
    count_launch();
    return L.z;
  }
  DLevel<TM>& C = H.lv[l + 1];
  if (s->mg_fused) {
    // this level and every coarser one in one block, when it is small enough
    if (n <= (size_t)MG_BLOCK_CELLS && H.lv.size() - l <= (size_t)MG_BLOCK_LEVELS) {
      MgChain<TM> m{};
      m.count = (int)(H.lv.size() - l);
      m.total = 0;
      for (int q = 0; q < m.count; ++q) {
        m.lv[q] = H.lv[l + q];
        m.off[q] = m.total;
        m.total += H.lv[l + q].w * H.lv[l + q].h;
      }
      const size_t smem = (size_t)7 * m.total * sizeof(TM);
      const DLevel<TM>& last = H.lv.back();
      if (smem <= 200 * 1024 && last.w * last.h <= 128) {
        if (kind == DT_CYCLE_JACOBI)
          k_mg_coarse<TM, true><<<1, 1024, smem, st>>>(m, NU, COARSE_SWEEPS);
        else
          k_mg_coarse<TM, false><<<1, 1024, smem, st>>>(m, NU, COARSE_SWEEPS_GS);
        count_launch();
        return L.z;
      }
    }
    // both sweeps of the smoothing in one launch over tiles, the restriction fused into the
    // pre-smoothing (the Gauss-Seidel cycle on two-colour levels)
    const bool jacobi = kind == DT_CYCLE_JACOBI;
    if (NU == 2 && tile_fits(L) && (jacobi || gs_colours(L.w, L.wrap) == 2)) {
      if (jacobi)
        launch_tile<TM, false, true>(s, L, C, nullptr, L.z, st);
      else
        launch_tile<TM, true, true>(s, L, C, nullptr, L.z, st);
      TM* zc = vcycle<TM>(s, H, l + 1, kind, st);
      if (jacobi)
        launch_tile<TM, false, false>(s, L, C, zc, L.t, st, rz);
      else
        launch_tile<TM, true, false>(s, L, C, zc, L.t, st, rz);
      return L.t;  // the level's z, in its spare buffer
    }
  }
  if (kind == DT_CYCLE_JACOBI) {
    // multigrid.rs:514-522
    TM *cur = L.z, *nxt = L.t;
    k_mg_first<TM><<<g, 256, 0, st>>>(L, cur);
    count_launch();
    for (int k = 1; k < NU; ++k) {
      k_mg_sweep<TM><<<g, 256, 0, st>>>(L, cur, nxt, nullptr, 0);
      count_launch();
      std::swap(cur, nxt);
    }
    k_mg_restrict<TM><<<dgrid(s, (size_t)C.w * C.h), 256, 0, st>>>(L, cur, C);
    count_launch();
    TM* zc = vcycle<TM>(s, H, l + 1, kind, st);
    k_mg_sweep<TM><<<g, 256, 0, st>>>(L, cur, nxt, zc, C.w);
    count_launch();
    std::swap(cur, nxt);
    for (int k = 1; k < NU; ++k) {
      k_mg_sweep<TM><<<g, 256, 0, st>>>(L, cur, nxt, nullptr, 0);
      count_launch();
      std::swap(cur, nxt);
    }
    return cur;
  }
  // multi-colour Gauss-Seidel V(NU, NU): colours forward, coarse correction, colours backward
  int ncol = gs_colours(L.w, L.wrap);
  for (int sweep = 0; sweep < NU; ++sweep)
    for (int c = 0; c < ncol; ++c) {
      if (sweep == 0)
        k_mg_gs<TM, true><<<g, 256, 0, st>>>(L, L.z, c);
      else
        k_mg_gs<TM, false><<<g, 256, 0, st>>>(L, L.z, c);
      count_launch();
    }
  k_mg_restrict<TM><<<dgrid(s, (size_t)C.w * C.h), 256, 0, st>>>(L, L.z, C);
  count_launch();
  TM* zc = vcycle<TM>(s, H, l + 1, kind, st);
  k_mg_prolong<TM><<<g, 256, 0, st>>>(L, L.z, zc, C.w);
  count_launch();
  for (int sweep = 0; sweep < NU; ++sweep)
    for (int c = ncol - 1; c >= 0; --c) {
      k_mg_gs<TM, false><<<g, 256, 0, st>>>(L, L.z, c);
      count_launch();
    }
  return L.z;
}

// The CG of one lane: vectors x, r, p, ap in TC; the cycle in TM on the levels of H; rm = H's
// finest r. Coefficients of the operator in TC.
template <class TC, class TM>
struct CgLane {
  TC *x, *r, *p, *ap, *east, *south, *diag;
  Hier<TM>* H;
  DScalars* S;
  TM* z;  // where the cycle leaves its result (set when the launch sequence is built)
};

// z = M^-1 r by one cycle, and r . z
template <class TC, class TM>
static TM* cycle_rz(dt_diff* s, CgLane<TC, TM>& C, int kind, cudaStream_t st) {
  RzArg rz{C.S, false};
  TM* z = vcycle<TM>(s, *C.H, 0, kind, st, std::is_same<TC, float>::value ? &rz : nullptr);
  if (!rz.done) {
    k_d_rz<TC, TM><<<dgrid(s, s->n), 256, 0, st>>>(s->n, C.r, z, s->partials, C.S);
    count_launch();
  }
  return z;
}

// The residual replacement of a reliable-update iteration (the FP32 lane): gated kernels that do
// nothing unless the iteration's update asked for it. `count`: count their launches (not inside
// the loop body's IF node, whose runs are counted from the replacements).
static void launch_reliable_d(dt_diff* s, cudaStream_t st, bool count) {
  unsigned int g = dgrid(s, s->n);
  k_d_rel_accumulate<<<g, 256, 0, st>>>(s->n, s->x, s->x32, s->scale, s->S32);
  k_d_apply<double, float, DA_RESID_GATED><<<g, 256, 0, st>>>(s->w, s->h, s->wrap && s->w > 1, s->east, s->south, s->diag, s->x,
                                                              s->b, s->r, nullptr, s->partials, s->S32);
  k_d_rel_reset<<<g, 256, 0, st>>>(s->n, s->r, s->r32, s->scale, s->S32);
  if (count)
    for (int k = 0; k < 3; ++k) count_launch();
}

// While `st` captures a loop body: a conditional IF node, its body the residual replacement
// (captured on `aside`), so that iterations that replace nothing launch nothing for it.
static dt_status add_reliable_if_d(dt_diff* s, cudaStream_t st, cudaStream_t aside, unsigned long long* handle_out) {
  cudaStreamCaptureStatus cs;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  DT_CUDA(cudaStreamGetCaptureInfo(st, &cs, &id, &graph, &deps, &nd));
  if (cs != cudaStreamCaptureStatusActive || !graph) {
    set_error("diffusion loop graph: the stream is not capturing");
    return DT_DEVICE_ERROR;
  }
  cudaGraphConditionalHandle h;
  DT_CUDA(cudaGraphConditionalHandleCreate(&h, graph, 0, cudaGraphCondAssignDefault));
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeIf;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  DT_CUDA(cudaGraphAddNode(&node, graph, deps, nd, &cp));
  DT_CUDA(cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
  DT_CUDA(cudaStreamBeginCaptureToGraph(aside, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal));
  launch_reliable_d(s, aside, false);
  cudaGraph_t ifbody;
  DT_CUDA(cudaStreamEndCapture(aside, &ifbody));
  *handle_out = (unsigned long long)h;
  return DT_OK;
}

// One CG iteration (multigrid.rs:698-733). With `reliable` (the FP32 lane of
// DT_DIFF_MIXED_RELIABLE) the residual replacement follows the update: under an IF node when
// `aside` is given (capturing a loop body; its handle goes to *if_handle), else launched gated.
template <class TC, class TM>
static dt_status cg_iteration(dt_diff* s, CgLane<TC, TM>& C, int kind, cudaStream_t st, bool reliable = false,
                              cudaStream_t aside = nullptr, unsigned long long* if_handle = nullptr) {
  unsigned int g = dgrid(s, s->n);
  k_d_apply<TC, TM, DA_PAP><<<g, 256, 0, st>>>(s->w, s->h, s->wrap && s->w > 1, C.east, C.south, C.diag, C.p, nullptr, C.ap,
                                                nullptr, s->partials, C.S);
  count_launch();
  k_d_update<TC, TM><<<g, 256, 0, st>>>(s->n, C.x, C.r, std::is_same<TC, TM>::value ? nullptr : C.H->lv[0].r, C.p, C.ap,
                                        s->partials, C.S);
  count_launch();
  if constexpr (std::is_same<TM, float>::value) {
    if (reliable) {
      if (aside)
        DT_TRY(add_reliable_if_d(s, st, aside, if_handle));
      else
        launch_reliable_d(s, st, true);
    }
  }
  TM* z = cycle_rz<TC, TM>(s, C, kind, st);
  C.z = z;
  k_d_direction<TC, TM><<<g, 256, 0, st>>>(s->n, C.p, z, C.S, 0);
  count_launch();
  return DT_OK;
}

template <class TC, class TM>
static dt_status cg_graph(dt_diff* s, CgLane<TC, TM>& C, int lane, int kind, DGraph** out, bool reliable = false) {
  DGraph& G = s->graph[lane][kind];
  if (G.exec) {
    *out = &G;
    return DT_OK;
  }
  cudaGraph_t g;
  DT_CUDA(cudaGraphCreate(&g, 0));
  cudaGraphConditionalHandle handle;
  DT_CUDA(cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault));
  unsigned long long hv = (unsigned long long)handle, hv_if = 0ull;
  DScalars* Sp = C.S;
  cudaKernelNodeParams kp = {};
  void* arm_args[] = {&Sp, &hv, &hv_if};
  kp.func = (void*)k_d_arm;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(1);
  kp.kernelParams = arm_args;
  cudaGraphNode_t n_arm, n_loop, n_disarm;
  DT_CUDA(cudaGraphAddKernelNode(&n_arm, g, nullptr, 0, &kp));
  cudaGraphNodeParams cp = {};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = handle;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  DT_CUDA(cudaGraphAddNode(&n_loop, g, &n_arm, 1, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  cudaStream_t aside = nullptr;
  if (reliable) DT_CUDA(cudaStreamCreateWithFlags(&aside, cudaStreamNonBlocking));
  DT_CUDA(cudaStreamBeginCaptureToGraph(s->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  begin_capture_count();
  dt_status st_body = cg_iteration<TC, TM>(s, C, kind, s->stream, reliable, aside, &hv_if);
  G.body_kernels = end_capture_count();
  cudaGraph_t captured;
  cudaError_t e_end = cudaStreamEndCapture(s->stream, &captured);
  if (aside) cudaStreamDestroy(aside);
  DT_TRY(st_body);
  DT_CUDA(e_end);
  if (reliable) DT_CUDA(cudaGraphKernelNodeSetParams(n_arm, &kp));  // k_d_arm learns the IF node's handle
  void* dis_args[] = {&Sp};
  kp.func = (void*)k_d_disarm;
  kp.kernelParams = dis_args;
  DT_CUDA(cudaGraphAddKernelNode(&n_disarm, g, &n_loop, 1, &kp));
  DT_CUDA(cudaGraphInstantiate(&G.exec, g, 0));
  G.g = g;
  *out = &G;
  return DT_OK;
}

static dt_status dread(dt_diff* s, const DScalars* S, DScalars* out) {
  DT_CUDA(cudaMemcpyAsync(out, S, sizeof(DScalars), cudaMemcpyDeviceToHost, s->stream));
  DT_CUDA(cudaStreamSynchronize(s->stream));
  return DT_OK;
}

// CG of lane C from x with r = b - A x, rm and S->rr, S->bb already set.
template <class TC, class TM>
static dt_status run_cg(dt_diff* s, CgLane<TC, TM>& C, int lane, int kind, const DProblem& prob, int host_loop, DScalars* out,
                        bool reliable = false) {
  cudaStream_t st = s->stream;
  unsigned int g = dgrid(s, s->n);
  k_d_begin<<<1, 1, 0, st>>>(C.S, prob, 0);
  count_launch();
  // the first direction: z = M^-1 r, rz, p = z
  TM* z = cycle_rz<TC, TM>(s, C, kind, st);
  k_d_direction<TC, TM><<<g, 256, 0, st>>>(s->n, C.p, z, C.S, 1);
  count_launch();
  if (!host_loop) {
    DGraph* G;
    DT_TRY(cg_graph<TC, TM>(s, C, lane, kind, &G, reliable));
    DT_CUDA(cudaGraphLaunch(G->exec, st));
    DT_TRY(dread(s, C.S, out));
    add_launches(2 + G->body_kernels * (long long)out->body_runs);
    return DT_OK;
  }
  DT_TRY(dread(s, C.S, out));
  for (int pass = 0; pass < prob.max_it + 2 && out->stop == DSTOP_RUNNING; ++pass) {
    DT_TRY(cg_iteration<TC, TM>(s, C, kind, st, reliable));
    DT_CUDA(cudaGetLastError());
    DT_TRY(dread(s, C.S, out));
    if (host_loop > 1)
      fprintf(stderr, "diffusion cg it %d stop %d rr %.6e rz %.6e alpha %.6e beta %.6e\n", out->it, out->stop, out->rr, out->rz,
              out->alpha, out->beta);
  }
  return DT_OK;
}

// Chunks of a segment of a line, and lines a block: columns in segments of 64 chunks (8 columns a
// block, or more of fewer chunks), rows of up to 512.
static void lod_shape(bool rows, int n, int* Pb, int* G, int* segments) {
  const int P = (int)ceil_div(n, LOD_CH), most = rows ? LOD_THREADS : LOD_THREADS / 8;
  *Pb = std::min(P, most);
  *G = std::max(1, std::min(LOD_THREADS / *Pb, rows ? LOD_THREADS : 32));
  *segments = (int)ceil_div(P, *Pb);
}
// L lines of n unknowns: b (the raster, or x itself) into s->x.
template <bool ROWS>
static void lod_lines(dt_diff* s, int L, int n, double dtdx2, const double* b) {
  cudaStream_t st = s->stream;
  int Pb, G, segments;
  lod_shape(ROWS, n, &Pb, &G, &segments);
  const dim3 grid(ceil_div(L, G), segments);
  const int threads = (int)ceil_div(Pb * G, 32) * 32;
  const size_t smem = lod_smem(ROWS);
  if (segments == 1) {
    k_lod_lines<ROWS, 0><<<grid, threads, smem, st>>>(L, n, Pb, G, dtdx2, s->kd, b, s->x, nullptr, nullptr);
    count_launch();
    return;
  }
  double* edge = s->lod[6];
  double* al = edge + (size_t)8 * segments * L;
  double* fact = al + (size_t)4 * segments * L;
  k_lod_lines<ROWS, 1><<<grid, threads, smem, st>>>(L, n, Pb, G, dtdx2, s->kd, b, s->x, edge, nullptr);
  k_lod_reduce<ROWS><<<ceil_div(L, 128), 128, 0, st>>>(L, n, segments, dtdx2, s->kd, edge, al, fact);
  k_lod_lines<ROWS, 2><<<grid, threads, smem, st>>>(L, n, Pb, G, dtdx2, s->kd, b, s->x, edge, fact);
  for (int k = 0; k < 3; ++k) count_launch();
}
static void lod_attributes() {
  cudaFuncSetAttribute(k_lod_lines<true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(true));
  cudaFuncSetAttribute(k_lod_lines<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(true));
  cudaFuncSetAttribute(k_lod_lines<true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(true));
  cudaFuncSetAttribute(k_lod_lines<false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(false));
  cudaFuncSetAttribute(k_lod_lines<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(false));
  cudaFuncSetAttribute(k_lod_lines<false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lod_smem(false));
}

static dt_status diff_first_guess(dt_diff* s, const dt_diff_params* p, double dt) {
  cudaStream_t st = s->stream;
  if (!p->first_guess) {
    DT_CUDA(cudaMemcpyAsync(s->x, s->b, s->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    return DT_OK;
  }
  const double dtdx2 = dt / (s->dx * s->dx);
  if (s->wrap && s->w > 2) {
    lod_lines<true>(s, s->h, s->w, dtdx2, s->b);
  } else {
    DT_CUDA(cudaMemcpyAsync(s->x, s->b, s->n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    k_lod_rows<<<ceil_div(s->h, 64), 64, 0, st>>>(s->w, s->h, s->wrap, s->x, s->kd, dtdx2, s->lod[0], s->lod[1], s->lod[2],
                                                  s->lod[3], s->lod[4], s->lod[5]);
    count_launch();
  }
  lod_lines<false>(s, s->w, s->h, dtdx2, s->x);
  return DT_OK;
}

template <class TM>
static Hier<TM>& hier_for(dt_diff* s, int kind);
template <>
Hier<float>& hier_for<float>(dt_diff* s, int kind) {
  return s->hf[kind];
}
template <>
Hier<double>& hier_for<double>(dt_diff* s, int kind) {
  return s->hd[kind];
}

// FP64 CG with a TM cycle (lane 0: TM = float, the reference's split; lane 1: TM = double).
template <class TM>
static dt_status solve_fp64_cg(dt_diff* s, const dt_diff_params* p, int lane, dt_report* rep, DScalars* fin) {
  cudaStream_t st = s->stream;
  Hier<TM>& H = hier_for<TM>(s, p->cycle);
  DT_TRY(build_levels<TM>(s, H, p->cycle == DT_CYCLE_JACOBI ? COARSEST : COARSEST_GS));
  fill_levels<TM>(s, H, p->cycle, st);
  unsigned int g = dgrid(s, s->n);
  int wrap = s->wrap && s->w > 1;
  // bb, then r = b - A x, rm, rr
  k_d_dot<double><<<g, 256, 0, st>>>(s->n, s->b, s->b, s->partials, s->S64);
  k_d_begin<<<1, 1, 0, st>>>(s->S64, DProblem{p->tol, p->max_iterations, p->stop, (int)s->n}, 1);
  k_d_apply<double, TM, DA_RESID><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->x, s->b, s->r,
                                                     std::is_same<TM, double>::value ? nullptr : H.lv[0].r,
                                                     s->partials, s->S64);
  count_launch();
  count_launch();
  count_launch();
  CgLane<double, TM> C{s->x, s->r, s->p, s->ap, s->east, s->south, s->diag, &H, s->S64, nullptr};
  DT_TRY(run_cg<double, TM>(s, C, lane, p->cycle, DProblem{p->tol, p->max_iterations, p->stop, (int)s->n}, p->host_loop, fin));
  if (rep) rep->iterations = fin->it;
  return DT_OK;
}

// FP32 inner CG (FP32 cycle) inside FP64 refinement on the residual scaled to unit RMS.
static dt_status solve_mixed_cg(dt_diff* s, const dt_diff_params* p, dt_report* rep, DScalars* fin) {
  cudaStream_t st = s->stream;
  Hier<float>& H = s->hf[p->cycle];
  DT_TRY(build_levels<float>(s, H, p->cycle == DT_CYCLE_JACOBI ? COARSEST : COARSEST_GS));
  fill_levels<float>(s, H, p->cycle, st);
  unsigned int g = dgrid(s, s->n);
  int wrap = s->wrap && s->w > 1;
  k_d_dot<double><<<g, 256, 0, st>>>(s->n, s->b, s->b, s->partials, s->S64);
  k_d_begin<<<1, 1, 0, st>>>(s->S64, DProblem{p->tol, p->max_iterations, p->stop, (int)s->n}, 1);
  count_launch();
  count_launch();
  int iterations = 0, refinements = 0;
  DScalars h64, h32;
  h32.stop = DSTOP_RUNNING;
  bool nonfinite = false;
  for (;;) {
    k_d_apply<double, float, DA_RESID><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->x, s->b, s->r, s->r32,
                                                          s->partials, s->S64);
    count_launch();
    DT_TRY(dread(s, s->S64, &h64));
    if (!std::isfinite(h64.rr) || !std::isfinite(h64.bb)) {
      nonfinite = true;
      break;
    }
    double lim2 = p->stop == DT_STOP_REL_RESIDUAL ? p->tol * p->tol * h64.bb : p->tol * p->tol * (double)s->n;
    if (h64.rr <= lim2) break;
    if (refinements >= p->max_refinements || iterations >= p->max_iterations) break;
    double rel = std::sqrt(h64.rr / std::max(lim2, 1e-300));  // > 1: how far above the target
    double itol = std::min(0.5, std::max(p->inner_tol, 0.3 / rel));
    k_d_scale_down<<<g, 256, 0, st>>>(s->n, s->r, s->r32, s->x32, s->S64, s->scale);
    // the inner system's b is the scaled residual: bb = its r.r, x = 0
    k_d_dot<float><<<g, 256, 0, st>>>(s->n, s->r32, s->r32, s->partials, s->S32);
    k_d_begin<<<1, 1, 0, st>>>(s->S32, DProblem{itol, p->max_iterations - iterations, DT_STOP_REL_RESIDUAL, (int)s->n}, 1);
    k_d_rr_is_bb<<<1, 1, 0, st>>>(s->S32);
    count_launch();
    count_launch();
    count_launch();
    count_launch();
    CgLane<float, float> C{s->x32, s->r32, s->p32, s->ap32, s->east32, s->south32, s->diag32, &H, s->S32, nullptr};
    DT_TRY(run_cg<float, float>(s, C, 2, p->cycle, DProblem{itol, p->max_iterations - iterations, DT_STOP_REL_RESIDUAL, (int)s->n},
                                p->host_loop, &h32));
    k_d_accumulate<<<g, 256, 0, st>>>(s->n, s->x, s->x32, s->scale);
    count_launch();
    iterations += h32.it;
    ++refinements;
    if (h32.stop == DSTOP_NONFINITE) {
      nonfinite = true;
      break;
    }
  }
  *fin = h64;
  fin->it = iterations;
  fin->stop = nonfinite ? DSTOP_NONFINITE
                        : (h64.rr <= (p->stop == DT_STOP_REL_RESIDUAL ? p->tol * p->tol * h64.bb : p->tol * p->tol * (double)s->n)
                               ? DSTOP_CONVERGED
                               : DSTOP_CAP);
  if (rep) {
    rep->iterations = iterations;
    rep->refinements = refinements;
  }
  return DT_OK;
}

// One FP32 CG (FP32 cycle) with reliable updates: the residual scaled to unit RMS once, then
// replaced by the FP64 b - A x (x folded into the FP64 accumulation) each time the FP32 residual
// has fallen a hundredfold or meets the tolerance; the FP64 residual alone decides convergence, and the
// search direction carries on, so the Krylov space is never restarted.
static dt_status solve_mixed_reliable(dt_diff* s, const dt_diff_params* p, dt_report* rep, DScalars* fin) {
  cudaStream_t st = s->stream;
  Hier<float>& H = s->hf[p->cycle];
  DT_TRY(build_levels<float>(s, H, p->cycle == DT_CYCLE_JACOBI ? COARSEST : COARSEST_GS));
  fill_levels<float>(s, H, p->cycle, st);
  unsigned int g = dgrid(s, s->n);
  int wrap = s->wrap && s->w > 1;
  k_d_dot<double><<<g, 256, 0, st>>>(s->n, s->b, s->b, s->partials, s->S64);
  k_d_begin<<<1, 1, 0, st>>>(s->S64, DProblem{p->tol, p->max_iterations, p->stop, (int)s->n}, 1);
  k_d_apply<double, float, DA_RESID><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->x, s->b, s->r, s->r32,
                                                        s->partials, s->S64);
  k_d_scale_down<<<g, 256, 0, st>>>(s->n, s->r, s->r32, s->x32, s->S64, s->scale);
  // replace when the FP32 residual has fallen a hundredfold: the V-cycle cuts it more than
  // tenfold an iteration, so a tenfold trigger would replace it every iteration
  k_d_rel_init<<<1, 1, 0, st>>>(s->S32, s->S64, s->scale, 0.01, p->stop == DT_STOP_RMS_RESIDUAL);
  for (int k = 0; k < 6; ++k) count_launch();
  CgLane<float, float> C{s->x32, s->r32, s->p32, s->ap32, s->east32, s->south32, s->diag32, &H, s->S32, nullptr};
  DScalars h32;
  DT_TRY(run_cg<float, float>(s, C, 3, p->cycle, DProblem{p->tol, p->max_iterations, DT_STOP_REL_RESIDUAL, (int)s->n, 1},
                              p->host_loop, &h32, true));
  if (!p->host_loop) add_launches(3LL * h32.replacements);
  // the correction since the last replacement (zero when the solve ended on one)
  k_d_accumulate<<<g, 256, 0, st>>>(s->n, s->x, s->x32, s->scale);
  count_launch();
  *fin = h32;
  if (rep) {
    rep->iterations = h32.it;
    rep->refinements = h32.replacements;
  }
  return DT_OK;
}

}  // namespace dt

using namespace dt;

extern "C" {

void dt_diff_default_params(dt_diff_params* p) {
  if (!p) return;
  p->cycle = DT_CYCLE_JACOBI;
  p->precision = DT_DIFF_FP64_CG_FP32_CYCLE;
  p->stop = DT_STOP_RMS_RESIDUAL;
  p->tol = 1e-5;             // surface.numerics.diffusion_tol_m (params.rs:197-200)
  p->max_iterations = 400;   // CG_MAX_ITER (diffusion.rs:497)
  p->first_guess = 1;        // the LOD splitting (diffusion.rs:101-110)
  p->inner_tol = 1e-5;
  p->max_refinements = 8;
  p->host_loop = 0;
}

dt_status dt_diff_destroy(dt_diff* s) {
  if (!s) return DT_OK;
  if (s->stream) cudaStreamSynchronize(s->stream);
  for (auto& a : s->graph)
    for (auto& G : a) {
      if (G.exec) cudaGraphExecDestroy(G.exec);
      if (G.g) cudaGraphDestroy(G.g);
    }
  for (void* q : s->allocs) cudaFree(q);
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  if (s->own_stream && s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return DT_OK;
}

dt_status dt_diff_create(int w, int h, double dx, int wrap_x, dt_diff** out) {
  if (!out) {
    set_error("dt_diff_create: out is NULL");
    return DT_BAD_ARG;
  }
  *out = nullptr;
  if (w < 1 || h < 1 || !(dx > 0.0) || !std::isfinite(dx)) {
    set_error("dt_diff_create: bad raster %d x %d, dx %g", w, h, dx);
    return DT_BAD_ARG;
  }
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    set_error("dt_diff_create: no CUDA device");
    return DT_DEVICE_ERROR;
  }
  auto* s = new dt_diff();
  s->w = w;
  s->h = h;
  s->dx = dx;
  s->wrap = wrap_x ? 1 : 0;
  if (const char* e = getenv("DT_MG_FUSED")) s->mg_fused = e[0] != '0';
  // the one-block coarse cycle stages at most about 4/3 MG_BLOCK_CELLS cells (plus the levels'
  // rounding up) in seven arrays
  cudaFuncSetAttribute(k_mg_coarse<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  cudaFuncSetAttribute(k_mg_coarse<double, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  cudaFuncSetAttribute(k_mg_coarse<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  cudaFuncSetAttribute(k_mg_coarse<double, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (const char* e = getenv("DT_MG_BIG_TILES")) s->mg_big_tiles = e[0] != '0';
  s->n = (size_t)w * h;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, 0) == cudaSuccess) s->sms = prop.multiProcessorCount;
  auto fail = [&](dt_status e) {
    dt_diff_destroy(s);
    return e;
  };
  if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(DT_DEVICE_ERROR);
  s->own_stream = true;
  dt_status st;
  for (double** q : {&s->kd, &s->b, &s->x, &s->r, &s->p, &s->ap, &s->east, &s->south, &s->diag})
    if ((st = ddalloc(s, q, s->n)) != DT_OK) return fail(st);
  for (float** q : {&s->east32, &s->south32, &s->diag32, &s->x32, &s->r32, &s->p32, &s->ap32})
    if ((st = ddalloc(s, q, s->n)) != DT_OK) return fail(st);
  // the LOD's scratch: the serial rows' arrays where the rows do not wrap, and the segments' relations
  // (8 values, 4 of their recurrence's) and Sherman-Morrison factors of lines of several segments
  if (!(s->wrap && s->w > 2))
    for (int k = 0; k < 6; ++k)
      if ((st = ddalloc(s, &s->lod[k], s->n)) != DT_OK) return fail(st);
  {
    int Pb, G, rows, cols;
    lod_shape(true, s->w, &Pb, &G, &rows);
    lod_shape(false, s->h, &Pb, &G, &cols);
    const size_t need = std::max(rows > 1 ? ((size_t)12 * rows + 1) * s->h : 0, cols > 1 ? (size_t)12 * cols * s->w : 0);
    if (need && (st = ddalloc(s, &s->lod[6], need)) != DT_OK) return fail(st);
  }
  lod_attributes();
  // a reducing kernel's blocks: two values each of at most eight an SM, or one of each of
  // k_mg_tile's tiles (56 x 24 cells at the least)
  const size_t tiles = (size_t)ceil_div(s->w, 56) * ceil_div(s->h, 24);
  if ((st = ddalloc(s, &s->partials, std::max((size_t)s->sms * 8 * 2, tiles))) != DT_OK) return fail(st);
  if ((st = ddalloc(s, &s->scale, 1)) != DT_OK) return fail(st);
  if ((st = ddalloc(s, &s->S64, 1)) != DT_OK) return fail(st);
  if ((st = ddalloc(s, &s->S32, 1)) != DT_OK) return fail(st);
  cudaMemset(s->S64, 0, sizeof(DScalars));
  cudaMemset(s->S32, 0, sizeof(DScalars));
  if (cudaEventCreate(&s->ev0) != cudaSuccess || cudaEventCreate(&s->ev1) != cudaSuccess) return fail(DT_DEVICE_ERROR);
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    set_error("dt_diff_create: %s", cudaGetErrorString(e));
    return fail(DT_DEVICE_ERROR);
  }
  *out = s;
  return DT_OK;
}

dt_status dt_diff_set_stream(dt_diff* s, void* stream) {
  if (!s) return DT_BAD_ARG;
  cudaStreamSynchronize(s->stream);
  if (s->own_stream) cudaStreamDestroy(s->stream);
  if (stream) {
    s->stream = (cudaStream_t)stream;
    s->own_stream = false;
  } else {
    if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return DT_DEVICE_ERROR;
    s->own_stream = true;
  }
  return DT_OK;
}

static dt_status diff_check(const dt_diff_params* p, double dt) {
  if (!p) {
    set_error("diffusion solve: params is NULL");
    return DT_BAD_ARG;
  }
  if ((p->cycle != DT_CYCLE_JACOBI && p->cycle != DT_CYCLE_RBGS) || p->precision < 0 || p->precision > 3 ||
      (p->stop != DT_STOP_RMS_RESIDUAL && p->stop != DT_STOP_REL_RESIDUAL) || !(p->tol >= 0.0) || p->max_iterations < 0) {
    set_error("diffusion solve: bad parameters (cycle %d, precision %d, rule %d, tol %g)", p->cycle, p->precision, p->stop, p->tol);
    return DT_BAD_ARG;
  }
  if (!(dt > 0.0) || !std::isfinite(dt)) {
    set_error("diffusion solve: dt must be positive and finite (got %g)", dt);
    return DT_BAD_ARG;
  }
  return DT_OK;
}

// The solve on kd and b already on the device (the handle's buffers).
static dt_status diff_solve_loaded(dt_diff* s, double dt, const dt_diff_params* p, dt_report* rep) {
  cudaStream_t st = s->stream;
  long long l0 = launches_now();
  cudaEventRecord(s->ev0, st);
  double dtdx2 = dt / (s->dx * s->dx);
  k_d_coeffs<<<dgrid(s, s->n), 256, 0, st>>>(s->w, s->h, s->wrap && s->w > 1, s->kd, dtdx2, s->east, s->south, s->diag, s->east32,
                                             s->south32, s->diag32);
  count_launch();
  DT_TRY(diff_first_guess(s, p, dt));
  DScalars fin;
  memset(&fin, 0, sizeof fin);
  if (rep) memset(rep, 0, sizeof *rep);
  if (p->precision == DT_DIFF_MIXED) {
    DT_TRY(solve_mixed_cg(s, p, rep, &fin));
  } else if (p->precision == DT_DIFF_MIXED_RELIABLE) {
    DT_TRY(solve_mixed_reliable(s, p, rep, &fin));
  } else if (p->precision == DT_DIFF_FP64) {
    DT_TRY(solve_fp64_cg<double>(s, p, 1, rep, &fin));
  } else {
    DT_TRY(solve_fp64_cg<float>(s, p, 0, rep, &fin));
  }
  // mass put-back: sum x = sum b (multigrid.rs:736-761)
  unsigned int g = dgrid(s, s->n);
  int wrap = s->wrap && s->w > 1;
  k_d_apply<double, float, DA_MASS><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->x, s->b, nullptr, nullptr,
                                                       s->partials, s->S64);
  k_d_massfix<<<g, 256, 0, st>>>(s->n, s->x, s->diag, s->S64);
  // the answer's relative residual
  k_d_apply<double, float, DA_RESID><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->x, s->b, s->ap, s->r32,
                                                        s->partials, s->S64);
  count_launch();
  count_launch();
  count_launch();
  cudaEventRecord(s->ev1, st);
  DScalars h;
  DT_TRY(dread(s, s->S64, &h));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, s->ev0, s->ev1);
  if (rep) {
    rep->converged = fin.stop == DSTOP_CONVERGED;
    rep->rel_residual = h.bb > 0 ? std::sqrt(h.rr / h.bb) : 0.0;
    rep->error_m = std::sqrt(h.rr / (double)s->n);  // the RMS residual, m
    rep->device_ms = ms;
    rep->kernel_launches = launches_now() - l0;
  }
  if (fin.stop == DSTOP_NONFINITE || !std::isfinite(h.rr)) {
    set_error("diffusion solve: a non-finite value appeared");
    return DT_NONFINITE;
  }
  return fin.stop == DSTOP_CONVERGED ? DT_OK : DT_NOT_CONVERGED;
}

dt_status dt_diff_solve(dt_diff* s, double* h_inout, const double* kd, double dt, const dt_diff_params* p, dt_report* rep) {
  if (!s || !h_inout || !kd) {
    set_error("dt_diff_solve: NULL argument");
    return DT_BAD_ARG;
  }
  DT_TRY(diff_check(p, dt));
  size_t bytes = s->n * sizeof(double);
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, bytes, cudaMemcpyHostToDevice, s->stream));
  DT_CUDA(cudaMemcpyAsync(s->b, h_inout, bytes, cudaMemcpyHostToDevice, s->stream));
  dt_status st = diff_solve_loaded(s, dt, p, rep);
  if (st == DT_OK || st == DT_NOT_CONVERGED) {
    DT_CUDA(cudaMemcpyAsync(h_inout, s->x, bytes, cudaMemcpyDeviceToHost, s->stream));
    DT_CUDA(cudaStreamSynchronize(s->stream));
  }
  return st;
}

dt_status dt_diff_solve_dev(dt_diff* s, double* h_inout, const double* kd, double dt, const dt_diff_params* p, dt_report* rep) {
  if (!s || !h_inout || !kd) {
    set_error("dt_diff_solve_dev: NULL argument");
    return DT_BAD_ARG;
  }
  DT_TRY(diff_check(p, dt));
  size_t bytes = s->n * sizeof(double);
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, bytes, cudaMemcpyDeviceToDevice, s->stream));
  DT_CUDA(cudaMemcpyAsync(s->b, h_inout, bytes, cudaMemcpyDeviceToDevice, s->stream));
  dt_status st = diff_solve_loaded(s, dt, p, rep);
  if (st == DT_OK || st == DT_NOT_CONVERGED) {
    DT_CUDA(cudaMemcpyAsync(h_inout, s->x, bytes, cudaMemcpyDeviceToDevice, s->stream));
    DT_CUDA(cudaStreamSynchronize(s->stream));
  }
  return st;
}

dt_status dt_diff_operator(dt_diff* s, const double* kd, double dt, const double* x, double* y) {
  if (!s || !kd || !x || !y) {
    set_error("dt_diff_operator: NULL argument");
    return DT_BAD_ARG;
  }
  size_t bytes = s->n * sizeof(double);
  cudaStream_t st = s->stream;
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, bytes, cudaMemcpyHostToDevice, st));
  DT_CUDA(cudaMemcpyAsync(s->p, x, bytes, cudaMemcpyHostToDevice, st));
  int wrap = s->wrap && s->w > 1;
  k_d_coeffs<<<dgrid(s, s->n), 256, 0, st>>>(s->w, s->h, wrap, s->kd, dt / (s->dx * s->dx), s->east, s->south, s->diag, s->east32,
                                             s->south32, s->diag32);
  k_d_apply<double, float, DA_PLAIN><<<dgrid(s, s->n), 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->p, nullptr,
                                                                    s->ap, nullptr, s->partials, s->S64);
  DT_CUDA(cudaGetLastError());
  DT_CUDA(cudaMemcpyAsync(y, s->ap, bytes, cudaMemcpyDeviceToHost, st));
  DT_CUDA(cudaStreamSynchronize(st));
  return DT_OK;
}

// x = the LOD splitting's first guess from h (host arrays; diffusion.rs:370-489)
dt_status dt_diff_lod(dt_diff* s, const double* h, const double* kd, double dt, double* x) {
  if (!s || !h || !kd || !x || !(dt > 0.0)) {
    set_error("dt_diff_lod: bad argument");
    return DT_BAD_ARG;
  }
  size_t bytes = s->n * sizeof(double);
  cudaStream_t st = s->stream;
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, bytes, cudaMemcpyHostToDevice, st));
  DT_CUDA(cudaMemcpyAsync(s->b, h, bytes, cudaMemcpyHostToDevice, st));
  dt_diff_params p;
  dt_diff_default_params(&p);
  p.first_guess = 1;
  DT_TRY(diff_first_guess(s, &p, dt));
  DT_CUDA(cudaGetLastError());
  DT_CUDA(cudaMemcpyAsync(x, s->x, bytes, cudaMemcpyDeviceToHost, st));
  DT_CUDA(cudaStreamSynchronize(st));
  return DT_OK;
}

dt_status dt_diff_vcycle(dt_diff* s, const double* kd, double dt, int cycle, const double* r, float* z, int* levels) {
  if (!s || !kd || !r || !z || (cycle != DT_CYCLE_JACOBI && cycle != DT_CYCLE_RBGS)) {
    set_error("dt_diff_vcycle: bad argument");
    return DT_BAD_ARG;
  }
  size_t bytes = s->n * sizeof(double);
  cudaStream_t st = s->stream;
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, bytes, cudaMemcpyHostToDevice, st));
  DT_CUDA(cudaMemcpyAsync(s->r, r, bytes, cudaMemcpyHostToDevice, st));
  int wrap = s->wrap && s->w > 1;
  k_d_coeffs<<<dgrid(s, s->n), 256, 0, st>>>(s->w, s->h, wrap, s->kd, dt / (s->dx * s->dx), s->east, s->south, s->diag, s->east32,
                                             s->south32, s->diag32);
  Hier<float>& H = s->hf[cycle];
  DT_TRY(build_levels<float>(s, H, cycle == DT_CYCLE_JACOBI ? COARSEST : COARSEST_GS));
  fill_levels<float>(s, H, cycle, st);
  k_convert_dr<<<dgrid(s, s->n), 256, 0, st>>>(s->n, s->r, H.lv[0].r);
  float* zz = vcycle<float>(s, H, 0, cycle, st);
  DT_CUDA(cudaGetLastError());
  DT_CUDA(cudaMemcpyAsync(z, zz, s->n * sizeof(float), cudaMemcpyDeviceToHost, st));
  DT_CUDA(cudaStreamSynchronize(st));
  if (levels) *levels = (int)H.lv.size();
  return DT_OK;
}

// Benchmark support: the CG operator (with p.Ap) and the Gauss-Seidel cycle's two tiled sweep
// pairs on the finest level, each launch timed alone (CUDA events on the handle's stream) after
// a write of a buffer twice the L2, so that it reads its inputs from HBM; ms[k] the mean of
// `reps` launches, bytes[k] the launch's algorithmic bytes (each array read once, each output
// written once). Inputs: x and the levels' r from kd, the coarse correction zero.
dt_status dt_diff_profile_kernels(dt_diff* s, const double* kd, double dt, int reps, double* ms, double* bytes) {
  if (!s || !kd || !ms || !bytes || reps < 1 || !(dt > 0.0)) {
    set_error("dt_diff_profile_kernels: bad argument");
    return DT_BAD_ARG;
  }
  cudaStream_t st = s->stream;
  const size_t n = s->n;
  const int wrap = s->wrap && s->w > 1;
  DT_CUDA(cudaMemcpyAsync(s->kd, kd, n * sizeof(double), cudaMemcpyHostToDevice, st));
  k_d_coeffs<<<dgrid(s, n), 256, 0, st>>>(s->w, s->h, wrap, s->kd, dt / (s->dx * s->dx), s->east, s->south, s->diag, s->east32,
                                          s->south32, s->diag32);
  Hier<float>& HF = s->hf[DT_CYCLE_RBGS];
  Hier<double>& HD = s->hd[DT_CYCLE_RBGS];
  DT_TRY(build_levels<float>(s, HF, COARSEST_GS));
  DT_TRY(build_levels<double>(s, HD, COARSEST_GS));
  if (HF.lv.size() < 2 || gs_colours(HF.lv[0].w, HF.lv[0].wrap) != 2 || HF.lv[0].w < 42 || !tile_fits(HF.lv[0])) {
    set_error("dt_diff_profile_kernels: the finest level of a %d x %d raster does not take the tiled sweeps", s->w, s->h);
    return DT_UNSUPPORTED;
  }
  fill_levels<float>(s, HF, DT_CYCLE_RBGS, st);
  fill_levels<double>(s, HD, DT_CYCLE_RBGS, st);
  DT_CUDA(cudaMemcpyAsync(s->p, s->kd, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  k_convert_dr<<<dgrid(s, n), 256, 0, st>>>(n, s->kd, s->p32);
  k_convert_dr<<<dgrid(s, n), 256, 0, st>>>(n, s->kd, HF.lv[0].r);
  DT_CUDA(cudaMemcpyAsync(HD.lv[0].r, s->kd, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  DLevel<float> &F0 = HF.lv[0], &F1 = HF.lv[1];
  DLevel<double> &D0 = HD.lv[0], &D1 = HD.lv[1];
  const size_t nc = (size_t)F1.w * F1.h;
  DT_CUDA(cudaMemsetAsync(F1.z, 0, nc * sizeof(float), st));
  DT_CUDA(cudaMemsetAsync(D1.z, 0, nc * sizeof(double), st));
  const unsigned g = dgrid(s, n);
  auto one = [&](int k) {
    switch (k) {
      case 0:
        k_d_apply<double, float, DA_PAP><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east, s->south, s->diag, s->p, nullptr, s->ap,
                                                            nullptr, s->partials, s->S64);
        break;
      case 1:
        k_d_apply<float, float, DA_PAP><<<g, 256, 0, st>>>(s->w, s->h, wrap, s->east32, s->south32, s->diag32, s->p32, nullptr,
                                                           s->ap32, nullptr, s->partials, s->S32);
        break;
      case 2: launch_tile<float, true, true>(s, F0, F1, nullptr, F0.z, st); break;
      case 3: launch_tile<float, true, false>(s, F0, F1, F1.z, F0.t, st); break;
      case 4: launch_tile<double, true, true>(s, D0, D1, nullptr, D0.z, st); break;
      default: launch_tile<double, true, false>(s, D0, D1, D1.z, D0.t, st); break;
    }
  };
  // algorithmic bytes: the operator x, east, south, diag in and y out; the pre-smoothing r, diag,
  // 1/diag, east, south in, z and the coarse r out; the post-smoothing z, the coarse z, r, diag,
  // 1/diag, east, south in and z out
  const double nf = (double)n, ncd = (double)nc;
  const double algo[DT_DIFF_PROFILE_KERNELS] = {40 * nf, 20 * nf, 4 * (6 * nf + ncd), 4 * (7 * nf + ncd),
                                                8 * (6 * nf + ncd), 8 * (7 * nf + ncd)};
  const size_t flush_bytes = (size_t)256 << 20;
  void* flush = nullptr;
  DT_CUDA(cudaMalloc(&flush, flush_bytes));
  cudaEvent_t a = nullptr, b = nullptr;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  dt_status rc = DT_OK;
  for (int k = 0; k < DT_DIFF_PROFILE_KERNELS && rc == DT_OK; ++k) {
    k_d_profile_state<<<1, 1, 0, st>>>(s->S64);
    k_d_profile_state<<<1, 1, 0, st>>>(s->S32);
    one(k);  // warm
    double total = 0.0;
    for (int r = 0; r < reps; ++r) {
      cudaMemsetAsync(flush, r & 0xff, flush_bytes, st);
      cudaEventRecord(a, st);
      one(k);
      cudaEventRecord(b, st);
      cudaEventSynchronize(b);
      float t = 0.f;
      cudaEventElapsedTime(&t, a, b);
      total += t;
    }
    if (cudaGetLastError() != cudaSuccess) {
      set_error("dt_diff_profile_kernels: a launch failed");
      rc = DT_DEVICE_ERROR;
    }
    ms[k] = total / reps;
    bytes[k] = algo[k];
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaStreamSynchronize(st);
  cudaFree(flush);
  return rc;
}

}  // extern "C"
