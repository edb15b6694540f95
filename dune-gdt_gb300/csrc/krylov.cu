// Device-resident Krylov solvers behind ConstMatrixOperator::apply_inverse
// (operators/matrix-based.hh:131-159). The reference hands this to dune-istl through dune-xt-la
// (third-party, absent from the reference tree); the algorithms restated here are the published
// ones: preconditioned CG (Hestenes-Stiefel), BiCGStab (van der Vorst 1992), Jacobi and ILU(0).
//
// GB300 design: all scalars (rho, alpha, beta, omega, residual norms, iteration count, converged
// flag) live in device memory; every reduction finishes in the last block of its kernel (ticketed,
// fixed summation order: deterministic), so an iteration issues no host synchronisation. Iterations
// are captured into a CUDA graph in chunks of `check_every`; the host reads the converged flag once
// per chunk, and kernels of iterations past convergence return immediately. FP64 CG with Jacobi or
// no preconditioner instead runs all its iterations, where persistent_applies, in one persistent
// launch (k_pcg_resident, k_pcg_stream below).
// Mixed precision: FP32 inner CG (FP32 CSR values, FP32 vectors, FP32 Jacobi) inside FP64
// iterative refinement with an FP64 residual r = b - A x from the FP64 matrix.
#include <cfloat>
#include <cmath>
#include <type_traits>
#include <vector>

#include "exchange.cuh"

namespace gdt {

namespace {

constexpr int TH = 256;

struct KState {
  double rho, alpha, beta, omega, rr, rr0, tol2, hden;
  int iter, max_iter, converged, breakdown;
};

__device__ __forceinline__ bool stopped(const KState* st) { return entry_flag(&st->converged) != 0; }

// ---------------------------------------------------------------- generic pieces ---
// y = A x; optional dot(w, y) -> st->hden / alpha (mode 1: CG alpha = rho / (p.Ap); mode 2: BiCGStab
// alpha = rho / (rt.v); mode 3: two dots (t.s, t.t) -> omega)
template <int G, int PL, class T, int MODE>
__global__ void __launch_bounds__(TH) k_spmv(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                            const T* __restrict__ val, const T* __restrict__ x, T* __restrict__ y,
                                            const T* __restrict__ w, KState* st, double* partials,
                                            unsigned int* ticket) {
  if (stopped(st)) return;
  T a0 = T(0), a1 = T(0);
  if constexpr (MODE == 0) {
    for_rows_csr<G, PL, T>(n, rp, col, val, x, [&](int row, bool leader, T s) {
      if (leader) y[row] = s;
    });
    return;
  } else {
    // the dot partner of row `row` (x for CG's p.Ap, w otherwise) is prefetched with the row bounds
    for_rows_csr_w<G, PL, T>(n, rp, col, val, x, MODE == 1 ? x : w, [&](int row, bool leader, T s, T wr) {
      if (leader) {
        y[row] = s;
        if (MODE == 1 || MODE == 2) a0 = fma(wr, s, a0);
        if (MODE == 3) {
          a0 = fma(s, wr, a0);
          a1 = fma(s, s, a1);
        }
      }
    });
  }
  double v[2] = {double(a0), double(a1)};
  if (grid_reduce<2>(v, partials, ticket) && threadIdx.x == 0) {
    if (MODE == 1) {
      if (!(v[0] > 0.0) || !isfinite(v[0])) {
        st->breakdown = 1;
        st->converged = 1;
      }
      st->alpha = st->rho / v[0];
    } else if (MODE == 2) {
      if (v[0] == 0.0 || !isfinite(v[0])) {
        st->breakdown = 1;
        st->converged = 1;
      }
      st->alpha = st->rho / v[0];
    } else {
      if (v[1] == 0.0 || !isfinite(v[1])) {
        st->breakdown = 1;
        st->converged = 1;
      }
      st->omega = v[0] / v[1];
    }
  }
}

// q = A p on the SELL-32 copy with p.q -> alpha: the graph-form CG SpMV where the SELL schedule
// was tuned fastest inside the iteration (or pinned)
__global__ void __launch_bounds__(256) k_sell_spmv_cg(SellView A, const double* __restrict__ p,
                                                      double* __restrict__ q, KState* st, double* partials,
                                                      unsigned int* ticket) {
  if (stopped(st)) return;
  double a0 = 0.0;
  for_slices<true>(
      A, p,
      [&](int row, bool active, double s, double pr) {
        if (active) {
          q[row] = s;
          a0 = fma(pr, s, a0);
        }
      },
      p);
  double v[1] = {a0};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    if (!(v[0] > 0.0) || !isfinite(v[0])) {
      st->breakdown = 1;
      st->converged = 1;
    }
    st->alpha = st->rho / v[0];
  }
}

// r = b - A x, z = M^{-1} r (Jacobi if dinv, else z = r), p = z (CG start); rho = r.z, rr0 = r.r
template <int G, int PL, class T>
__global__ void __launch_bounds__(TH) k_residual_init(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                     const T* __restrict__ val, const T* __restrict__ x,
                                                     const T* __restrict__ b, T* __restrict__ r,
                                                     const T* __restrict__ dinv, T* __restrict__ p,
                                                     KState* st, double* partials, unsigned int* ticket) {
  T a0 = T(0), a1 = T(0);
  for_rows_csr<G, PL, T>(n, rp, col, val, x, [&](int row, bool leader, T s) {
    if (leader) {
      T ri = b[row] - s;
      r[row] = ri;
      T zi = dinv ? dinv[row] * ri : ri;
      if (p) p[row] = zi;
      a0 = fma(ri, zi, a0);
      a1 = fma(ri, ri, a1);
    }
  });
  double v[2] = {double(a0), double(a1)};
  if (grid_reduce<2>(v, partials, ticket) && threadIdx.x == 0) {
    st->rho = v[0];
    st->rr = v[1];
    st->rr0 = v[1];
    st->iter = 0;
    st->breakdown = 0;
    st->alpha = st->beta = st->omega = 1.0;
    st->converged = (v[1] == 0.0 || v[1] <= st->tol2 * v[1]) ? 1 : 0;
    if (!isfinite(v[1])) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

// x0 = 0 start of the inner FP32 solve: r holds b already; p = dinv r; rho = r.p, rr0 = r.r
template <class T>
__global__ void __launch_bounds__(TH) k_init_from_rhs(int n, const T* __restrict__ r, const T* __restrict__ dinv,
                                                     T* __restrict__ p, KState* st, double* partials,
                                                     unsigned int* ticket) {
  T a0 = T(0), a1 = T(0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    T ri = r[i];
    T zi = dinv[i] * ri;
    p[i] = zi;
    a0 = fma(ri, zi, a0);
    a1 = fma(ri, ri, a1);
  }
  double v[2] = {double(a0), double(a1)};
  if (grid_reduce<2>(v, partials, ticket) && threadIdx.x == 0) {
    st->rho = v[0];
    st->rr = v[1];
    st->rr0 = v[1];
    st->iter = 0;
    st->breakdown = 0;
    st->alpha = st->beta = st->omega = 1.0;
    st->converged = (v[1] == 0.0) ? 1 : 0;
  }
}

// CG with Jacobi, fused: x += alpha p; r -= alpha q; z = dinv r (not stored); rho' = r.z, rr = r.r
template <class TX, class T>
__global__ void __launch_bounds__(TH) k_cg_update_jacobi(int n, TX* __restrict__ x, const T* __restrict__ p,
                                                        T* __restrict__ r, const T* __restrict__ q,
                                                        const T* __restrict__ dinv, KState* st, double* partials,
                                                        unsigned int* ticket) {
  if (stopped(st)) return;
  const T alpha = T(st->alpha);
  T a0 = T(0), a1 = T(0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = TX(fma(alpha, p[i], T(x[i])));
    T ri = fma(-alpha, q[i], r[i]);
    r[i] = ri;
    a0 = fma(ri, dinv[i] * ri, a0);
    a1 = fma(ri, ri, a1);
  }
  double v[2] = {double(a0), double(a1)};
  if (grid_reduce<2>(v, partials, ticket) && threadIdx.x == 0) {
    st->beta = v[0] / st->rho;
    st->rho = v[0];
    st->rr = v[1];
    st->iter += 1;
    if (v[1] <= st->tol2 * st->rr0 || st->iter >= st->max_iter) st->converged = 1;
    if (!isfinite(v[1])) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

// The same two FP64 kernels on pairs of rows (16-byte loads and stores, twice the bytes in flight
// per instruction); for vectors that all start on a 16-byte boundary. The odd last row, if any, is
// done by the first thread of the grid.
__global__ void __launch_bounds__(TH) k_cg_update_jacobi2(int n, double* __restrict__ x, const double* __restrict__ p,
                                                         double* __restrict__ r, const double* __restrict__ q,
                                                         const double* __restrict__ dinv, KState* st,
                                                         double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  const double alpha = st->alpha;
  double a0 = 0.0, a1 = 0.0;
  const int n2 = n >> 1;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n2; k += gridDim.x * blockDim.x) {
    double2 xv = reinterpret_cast<const double2*>(x)[k], rv = reinterpret_cast<const double2*>(r)[k];
    const double2 pv = reinterpret_cast<const double2*>(p)[k], qv = reinterpret_cast<const double2*>(q)[k],
                  dv = reinterpret_cast<const double2*>(dinv)[k];
    xv.x = fma(alpha, pv.x, xv.x);
    xv.y = fma(alpha, pv.y, xv.y);
    rv.x = fma(-alpha, qv.x, rv.x);
    rv.y = fma(-alpha, qv.y, rv.y);
    a0 = fma(rv.x, dv.x * rv.x, a0);
    a1 = fma(rv.x, rv.x, a1);
    a0 = fma(rv.y, dv.y * rv.y, a0);
    a1 = fma(rv.y, rv.y, a1);
    reinterpret_cast<double2*>(x)[k] = xv;
    reinterpret_cast<double2*>(r)[k] = rv;
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const int i = n - 1;
    x[i] = fma(alpha, p[i], x[i]);
    const double ri = fma(-alpha, q[i], r[i]);
    r[i] = ri;
    a0 = fma(ri, dinv[i] * ri, a0);
    a1 = fma(ri, ri, a1);
  }
  double v[2] = {a0, a1};
  if (grid_reduce<2>(v, partials, ticket) && threadIdx.x == 0) {
    st->beta = v[0] / st->rho;
    st->rho = v[0];
    st->rr = v[1];
    st->iter += 1;
    if (v[1] <= st->tol2 * st->rr0 || st->iter >= st->max_iter) st->converged = 1;
    if (!isfinite(v[1])) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

__global__ void __launch_bounds__(TH) k_cg_p_jacobi2(int n, double* __restrict__ p, const double* __restrict__ r,
                                                    const double* __restrict__ dinv, const KState* st) {
  if (stopped(st)) return;
  const double beta = st->beta;
  const int n2 = n >> 1;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n2; k += gridDim.x * blockDim.x) {
    double2 pv = reinterpret_cast<const double2*>(p)[k];
    const double2 rv = reinterpret_cast<const double2*>(r)[k], dv = reinterpret_cast<const double2*>(dinv)[k];
    pv.x = fma(beta, pv.x, dv.x * rv.x);
    pv.y = fma(beta, pv.y, dv.y * rv.y);
    reinterpret_cast<double2*>(p)[k] = pv;
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) p[n - 1] = fma(beta, p[n - 1], dinv[n - 1] * r[n - 1]);
}

template <class T>
__global__ void __launch_bounds__(TH) k_cg_p_jacobi(int n, T* __restrict__ p, const T* __restrict__ r,
                                                   const T* __restrict__ dinv, const KState* st) {
  if (stopped(st)) return;
  const T beta = T(st->beta);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    p[i] = fma(beta, p[i], dinv[i] * r[i]);
}

// generic CG (any preconditioner): x += alpha p; r -= alpha q; rr = r.r
__global__ void __launch_bounds__(TH) k_cg_update(int n, double* __restrict__ x, const double* __restrict__ p,
                                                 double* __restrict__ r, const double* __restrict__ q, KState* st,
                                                 double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  const double alpha = st->alpha;
  double a0 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = fma(alpha, p[i], x[i]);
    double ri = fma(-alpha, q[i], r[i]);
    r[i] = ri;
    a0 = fma(ri, ri, a0);
  }
  double v[1] = {a0};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    st->rr = v[0];
    st->iter += 1;
    if (v[0] <= st->tol2 * st->rr0 || st->iter >= st->max_iter) st->converged = 1;
    if (!isfinite(v[0])) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

// rho' = r.z, beta = rho'/rho (CG)
__global__ void __launch_bounds__(TH) k_cg_beta(int n, const double* __restrict__ r, const double* __restrict__ z,
                                               KState* st, double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  double a0 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a0 = fma(r[i], z[i], a0);
  double v[1] = {a0};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    st->beta = v[0] / st->rho;
    st->rho = v[0];
  }
}

__global__ void __launch_bounds__(TH) k_cg_p(int n, double* __restrict__ p, const double* __restrict__ z,
                                            const KState* st) {
  if (stopped(st)) return;
  const double beta = st->beta;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = fma(beta, p[i], z[i]);
}

// ---------------------------------------------------------------- BiCGStab pieces ---
// rho' = rt.r ; beta = (rho'/rho)(alpha/omega) ; p = r + beta (p - omega v) (first iteration: p = r)
__global__ void __launch_bounds__(TH) k_bicg_rho(int n, const double* __restrict__ rt, const double* __restrict__ r,
                                                KState* st, double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  double a0 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a0 = fma(rt[i], r[i], a0);
  double v[1] = {a0};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    if (v[0] == 0.0 || !isfinite(v[0])) {
      st->breakdown = 1;
      st->converged = 1;
    }
    st->beta = (st->iter == 0) ? 0.0 : (v[0] / st->rho) * (st->alpha / st->omega);
    st->rho = v[0];
  }
}

__global__ void __launch_bounds__(TH) k_bicg_p(int n, double* __restrict__ p, const double* __restrict__ r,
                                              const double* __restrict__ v, const KState* st) {
  if (stopped(st)) return;
  const double beta = st->beta, omega = st->omega;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    p[i] = fma(beta, fma(-omega, v[i], p[i]), r[i]);
}

// x += alpha y ; s = r - alpha v ; check ||s|| (if converged: r = s)
__global__ void __launch_bounds__(TH) k_bicg_s(int n, double* __restrict__ x, const double* __restrict__ y,
                                              double* __restrict__ r, const double* __restrict__ v, KState* st,
                                              double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  const double alpha = st->alpha;
  double a0 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = fma(alpha, y[i], x[i]);
    double si = fma(-alpha, v[i], r[i]);
    r[i] = si;  // r now holds s
    a0 = fma(si, si, a0);
  }
  double w[1] = {a0};
  if (grid_reduce<1>(w, partials, ticket) && threadIdx.x == 0) {
    st->rr = w[0];
    if (w[0] <= st->tol2 * st->rr0) {
      st->iter += 1;
      st->converged = 1;
    }
  }
}

// x += omega z ; r = s - omega t ; rr
__global__ void __launch_bounds__(TH) k_bicg_r(int n, double* __restrict__ x, const double* __restrict__ z,
                                              double* __restrict__ r, const double* __restrict__ t, KState* st,
                                              double* partials, unsigned int* ticket) {
  if (stopped(st)) return;
  const double omega = st->omega;
  double a0 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    x[i] = fma(omega, z[i], x[i]);
    double ri = fma(-omega, t[i], r[i]);
    r[i] = ri;
    a0 = fma(ri, ri, a0);
  }
  double w[1] = {a0};
  if (grid_reduce<1>(w, partials, ticket) && threadIdx.x == 0) {
    st->rr = w[0];
    st->iter += 1;
    if (w[0] <= st->tol2 * st->rr0 || st->iter >= st->max_iter) st->converged = 1;
    if (!isfinite(w[0])) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

// ------------------------------------------------------------------- preconditioners ---
template <class TD, class TS>
__global__ void k_jacobi_diag(int n, const int* __restrict__ rp, const int* __restrict__ col,
                              const TS* __restrict__ val, TD* __restrict__ dinv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    TS d = TS(0);
    for (int k = rp[i]; k < rp[i + 1]; ++k)
      if (col[k] == i) d = val[k];
    dinv[i] = TD(1.0 / double(d));
  }
}

template <class T>
__global__ void k_scale(int n, T* __restrict__ z, const T* __restrict__ d, const T* __restrict__ r, const KState* st) {
  if (stopped(st)) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = d ? d[i] * r[i] : r[i];
}

// ILU(0), level scheduled: rows of one level depend only on rows of earlier levels.
__global__ void k_ilu_factor_level(const int* __restrict__ rows, int count, const int* __restrict__ rp,
                                   const int* __restrict__ col, const int* __restrict__ diag, double* __restrict__ lu) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t];
  const int end_i = rp[i + 1];
  for (int pk = rp[i]; pk < end_i; ++pk) {
    const int k = col[pk];
    if (k >= i) break;
    const double lik = lu[pk] / lu[diag[k]];
    lu[pk] = lik;
    int pi = pk + 1;
    for (int pj = diag[k] + 1; pj < rp[k + 1]; ++pj) {
      const int j = col[pj];
      while (pi < end_i && col[pi] < j) ++pi;
      if (pi < end_i && col[pi] == j) lu[pi] -= lik * lu[pj];
    }
  }
}

__global__ void k_ilu_lower_level(const int* __restrict__ rows, int count, const int* __restrict__ rp,
                                  const int* __restrict__ col, const int* __restrict__ diag,
                                  const double* __restrict__ lu, const double* __restrict__ r, double* __restrict__ z,
                                  const KState* st) {
  if (stopped(st)) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t];
  double s = r[i];
  for (int p = rp[i]; p < diag[i]; ++p) s -= lu[p] * z[col[p]];
  z[i] = s;
}

__global__ void k_ilu_upper_level(const int* __restrict__ rows, int count, const int* __restrict__ rp,
                                  const int* __restrict__ col, const int* __restrict__ diag,
                                  const double* __restrict__ lu, double* __restrict__ z, const KState* st) {
  if (stopped(st)) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  const int i = rows[t];
  double s = z[i];
  for (int p = diag[i] + 1; p < rp[i + 1]; ++p) s -= lu[p] * z[col[p]];
  z[i] = s / lu[diag[i]];
}

__global__ void k_find_diag(int n, const int* __restrict__ rp, const int* __restrict__ col, int* __restrict__ diag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int d = -1;
    for (int k = rp[i]; k < rp[i + 1]; ++k)
      if (col[k] == i) d = k;
    diag[i] = d;
  }
}

// -------------------------------------------------------------- mixed precision helpers ---
__global__ void k_to_float(long long n, const double* __restrict__ a, float* __restrict__ b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = float(a[i]);
}

// r64 = b - A x (FP64) ; rr = r.r ; r32 = r64 * inv_scale where inv_scale = 1/||r|| is applied on the host side
template <int G, int PL>
__global__ void __launch_bounds__(TH) k_residual64(int n, const int* __restrict__ rp, const int* __restrict__ col,
                                                  const double* __restrict__ val, const double* __restrict__ x,
                                                  const double* __restrict__ b, double* __restrict__ r,
                                                  double* out_rr, double* partials, unsigned int* ticket) {
  double a0 = 0.0;
  for_rows_csr<G, PL, double>(n, rp, col, val, x, [&](int row, bool leader, double s) {
    if (leader) {
      double ri = b[row] - s;
      r[row] = ri;
      a0 = fma(ri, ri, a0);
    }
  });
  double v[1] = {a0};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) *out_rr = v[0];
}

__global__ void k_scale_to_float(int n, const double* __restrict__ r, const double* __restrict__ rr,
                                 float* __restrict__ r32) {
  const double inv = 1.0 / sqrt(*rr);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) r32[i] = float(r[i] * inv);
}

__global__ void k_correct(int n, double* __restrict__ x, const float* __restrict__ d, const double* __restrict__ rr) {
  const double scale = sqrt(*rr);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    x[i] = fma(scale, double(d[i]), x[i]);
}

// ---------------------------------------------------------------------------- host ---
struct Launch {
  gdt_context ctx;
  int n;
  int sched;
  int vec_blocks;
  cudaStream_t s;
  double* partials;
  unsigned int* ticket;
  template <class T>
  LaunchShape shape() const {
    return schedule_shape<T>(sched, n, ctx->num_sms);
  }
};

// the graph-form CG SpMV (q = A p, alpha) on the SELL-32 copy
void spmv_cg_sell(const Launch& L, gdt_matrix m, const double* p, double* q, KState* st) {
  const SellView A = sell_view(m);
  timing_begin(L.ctx, L.s, GDT_TIMING_SPMV_FP64);
  k_sell_spmv_cg<<<sell_blocks(A.nslices, L.ctx->num_sms, reinterpret_cast<const void*>(&k_sell_spmv_cg)), 256, 0,
                   L.s>>>(A, p, q, st, L.partials, L.ticket);
  timing_end(L.ctx, L.s);
  L.ctx->launches++;
}

template <class T, int MODE>
void spmv_mode(const Launch& L, const int* rp, const int* col, const T* val, const T* x, T* y, const T* w,
               KState* st) {
  const LaunchShape sh = L.shape<T>();
  timing_begin(L.ctx, L.s, sizeof(T) == 8 ? GDT_TIMING_SPMV_FP64 : GDT_TIMING_SPMV_FP32);
#define GDT_K_SPMV(GG, PP) \
  k_spmv<GG, PP, T, MODE><<<sh.blocks, sh.threads, sh.smem, L.s>>>(L.n, rp, col, val, x, y, w, st, L.partials, L.ticket)
  GDT_SCHEDULE_SWITCH(L.sched, GDT_K_SPMV)
#undef GDT_K_SPMV
  timing_end(L.ctx, L.s);
  L.ctx->launches++;
}

template <class T>
void residual_init(const Launch& L, const int* rp, const int* col, const T* val, const T* x, const T* b, T* r,
                   const T* dinv, T* p, KState* st) {
  const LaunchShape sh = L.shape<T>();
#define GDT_K_RESINIT(GG, PP)                                                                                    \
  k_residual_init<GG, PP, T><<<sh.blocks, sh.threads, sh.smem, L.s>>>(L.n, rp, col, val, x, b, r, dinv, p, st, \
                                                                      L.partials, L.ticket)
  GDT_SCHEDULE_SWITCH(L.sched, GDT_K_RESINIT)
#undef GDT_K_RESINIT
  L.ctx->launches++;
}

void residual64(const Launch& L, gdt_matrix m, const double* x, const double* b, double* r, double* rr) {
  const LaunchShape sh = L.shape<double>();
#define GDT_K_RES64(GG, PP)                                                                                      \
  k_residual64<GG, PP><<<sh.blocks, sh.threads, sh.smem, L.s>>>(L.n, m->rp, m->col, m->val, x, b, r, rr, L.partials, \
                                                                L.ticket)
  GDT_SCHEDULE_SWITCH(L.sched, GDT_K_RES64)
#undef GDT_K_RES64
  L.ctx->launches++;
}

// level sets of the lower (U = false) or upper (U = true) triangle, computed on the host from the pattern
void level_sets(int n, const std::vector<int>& rp, const std::vector<int>& col, bool upper, std::vector<int>& order,
                std::vector<int>& offsets) {
  std::vector<int> lev(n, 0);
  int maxl = 0;
  if (!upper) {
    for (int i = 0; i < n; ++i) {
      int l = 0;
      for (int k = rp[i]; k < rp[i + 1] && col[k] < i; ++k) l = std::max(l, lev[col[k]] + 1);
      lev[i] = l;
      maxl = std::max(maxl, l);
    }
  } else {
    for (int i = n - 1; i >= 0; --i) {
      int l = 0;
      for (int k = rp[i + 1] - 1; k >= rp[i] && col[k] > i; --k) l = std::max(l, lev[col[k]] + 1);
      lev[i] = l;
      maxl = std::max(maxl, l);
    }
  }
  offsets.assign(maxl + 2, 0);
  for (int i = 0; i < n; ++i) offsets[lev[i] + 1]++;
  for (int l = 0; l <= maxl; ++l) offsets[l + 1] += offsets[l];
  order.resize(n);
  std::vector<int> fill(offsets.begin(), offsets.end() - 1);
  for (int i = 0; i < n; ++i) order[fill[lev[i]]++] = i;
}

struct Ilu {
  double* lu = nullptr;
  int* diag = nullptr;
  int* lorder = nullptr;
  int* uorder = nullptr;
  std::vector<int> loff, uoff;
};

gdt_status ilu_setup(gdt_context ctx, gdt_matrix m, Ilu& f, cudaStream_t s) {
  const int n = int(m->rows);
  std::vector<int> rp(n + 1), col(m->nnz);
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(rp.data(), m->rp, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(col.data(), m->col, sizeof(int) * m->nnz, cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  std::vector<int> lo, uo;
  level_sets(n, rp, col, false, lo, f.loff);
  level_sets(n, rp, col, true, uo, f.uoff);
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &f.lu, sizeof(double) * m->nnz, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &f.diag, sizeof(int) * n, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &f.lorder, sizeof(int) * n, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &f.uorder, sizeof(int) * n, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(f.lorder, lo.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(f.uorder, uo.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(f.lu, m->val, sizeof(double) * m->nnz, cudaMemcpyDeviceToDevice, s));
  k_find_diag<<<grid_blocks(n, TH), TH, 0, s>>>(n, m->rp, m->col, f.diag);
  GDT_CHECK(ctx, check_launch(ctx, "ilu diag"));
  for (size_t l = 0; l + 1 < f.loff.size(); ++l) {
    int cnt = f.loff[l + 1] - f.loff[l];
    k_ilu_factor_level<<<grid_blocks(cnt, 128), 128, 0, s>>>(f.lorder + f.loff[l], cnt, m->rp, m->col, f.diag, f.lu);
    GDT_CHECK(ctx, check_launch(ctx, "ilu factor"));
  }
  // keep the host copies alive until the asynchronous uploads have completed
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  return GDT_OK;
}

void ilu_apply(gdt_context ctx, gdt_matrix m, const Ilu& f, const double* r, double* z, const KState* st,
               cudaStream_t s) {
  for (size_t l = 0; l + 1 < f.loff.size(); ++l) {
    int cnt = f.loff[l + 1] - f.loff[l];
    k_ilu_lower_level<<<grid_blocks(cnt, 128), 128, 0, s>>>(f.lorder + f.loff[l], cnt, m->rp, m->col, f.diag, f.lu, r,
                                                            z, st);
    ctx->launches++;
  }
  for (size_t l = 0; l + 1 < f.uoff.size(); ++l) {
    int cnt = f.uoff[l + 1] - f.uoff[l];
    k_ilu_upper_level<<<grid_blocks(cnt, 128), 128, 0, s>>>(f.uorder + f.uoff[l], cnt, m->rp, m->col, f.diag, f.lu, z,
                                                            st);
    ctx->launches++;
  }
}


// ------------------------------------------------------------------------- persistent CG ---
// One cooperative launch runs every iteration of Jacobi-preconditioned (or plain) CG; two grid-wide
// sums per iteration take the place of the graph form's kernel boundaries.
//
// What bounds an iteration here is not bandwidth but the FP64 pipe (one warp instruction per 19 SM
// cycles) and the grid-wide waits, so the kernel is built around those two:
//  * The x, r and direction updates are one pass. beta needs rho' = r'.z', which classically waits for
//    a sum over the updated residual. With r' = r - alpha q it is rho - 2 alpha (z.q) + alpha^2 (q.D^-1 q),
//    and both products are summed together with p.q right after q = A p (cf. Meurant 1987). beta takes
//    that value; alpha and the stopping test take the sums over the residual itself, so nothing
//    accumulates: the iteration counts are those of the classical form, also on badly conditioned 1D
//    systems, where the shorter alpha^2 (q.D^-1 q) - rho (z.q = p.q) needs up to 38 % more.
//  * A grid-wide sum and the barrier it implies are one exchange (exchange.cuh), and the scalars
//    that follow, a reciprocal and a few products, are formed by one thread.
//  * A thread owns its rows for the whole solve: x, r, p, D^-1 and q of k_pcg_resident never leave its
//    registers (p is also written for the neighbours' gathers), and a block keeps as much of its
//    matrix as fits in shared memory.
//  * Entries that are exactly zero (the hypotenuse couplings of P1 on right-angled simplices, the
//    columns of Dirichlet rows) are dropped from the SELL-32 copy: no loads and no FMAs for them.
//  * Work is spread over all SMs, down to one 32-row slice per block.
// The matrix and D^-1 are read-only in the kernels (non-coherent loads); p is written by other blocks
// between the sums and read with plain loads, which the fences of the exchanges order.
struct PcgArgs {
  int n;
  const int2* meta;   // SELL-32 (offset, width) per slice
  const int* width;   // entries per row of the slice after dropping zeros
  const int* col;     // SELL-32 columns
  const double* val;  // SELL-32 values
  const double* dinv;
  double* x;
  double* r;
  double* p;
  double* q;
  KState* st;
  ExchangeView ex;    // the whole grid
  int cap;            // matrix entries a block may keep in shared memory (resident form)
  float keep;         // share of the matrix that L2 may keep; the rest is marked evict-first
  int qshared;        // the streaming form keeps q in shared memory
  int units;          // the most units of a block (streaming form by units)
  int short_rows;     // no row has more than three entries
  int first[257];     // the block's slices: first[block] .. first[block + 1] - 1
};

// The scalars of the iteration, kept by thread 0 of every block (the same bits in all of them).
struct PcgScalars {
  double rho, alpha, beta, rr, stop;
  int iter, max_iter, conv;
  int brk;  // 1: breakdown; 2: alpha or beta left the range of a double, the iterate before it is good
  __device__ void load(const KState* st) {
    rho = st->rho;
    alpha = st->alpha;
    beta = st->beta;
    rr = st->rr;
    stop = st->tol2 * st->rr0;
    iter = st->iter;
    max_iter = st->max_iter;
    conv = brk = 0;
  }
  __device__ void store(KState* st) const {
    st->rho = rho;
    st->alpha = alpha;
    st->beta = beta;
    st->rr = rr;
    st->iter = iter;
    st->breakdown = brk;
    st->converged = 1;
  }
};

template <int T>
struct PcgShared {
  ExchangeShared<T> ex;
  double total[3];
  double last[2];
  PcgScalars k;
  int go;
};

// on the integer pipe: thread 0 decides while the others wait
__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// v = (p.q, z.q, q.D^-1 q) over the rows of the thread: alpha and beta in sh.k; false when done. The stopping test
// of the iteration before is made here too: its sums (sh.last) are formed while the other warps
// already multiply, so a solve ends with one product it does not use.
template <bool CLUSTER, int T>
__device__ __forceinline__ bool pcg_step(const PcgArgs& a, unsigned int& epoch, const double (&v)[3], int warps,
                                         PcgShared<T>& sh) {
  const bool first = epoch == 0;
  double total;
  if constexpr (CLUSTER) total = cluster_exchange(epoch, v, warps, sh.ex);
  else total = group_exchange<false>(a.ex, epoch, v, warps, sh.ex);
  if (threadIdx.x < 96) {
    const double inv = threadIdx.x == 0 ? 1.0 / total : 0.0;
    if ((threadIdx.x & 31) == 0) sh.total[threadIdx.x >> 5] = total;
    asm volatile("bar.sync 1, 96;" ::: "memory");
    if (threadIdx.x == 0) {
      PcgScalars& k = sh.k;
      if (!first) {
        k.rho = sh.last[0];
        k.rr = sh.last[1];
        k.iter += 1;
        if (k.rr <= k.stop || k.iter >= k.max_iter) k.conv = 1;
        if (!finite_bits(k.rr)) k.brk = k.conv = 1;
      }
      if (!k.conv) {
        k.alpha = k.rho * inv;
        k.beta = fma(k.alpha * inv, sh.total[2], fma(-2.0 * inv, sh.total[1], 1.0));
        if (__double_as_longlong(total) <= 0 || !finite_bits(total)) k.brk = k.conv = 1;
        else if (!finite_bits(k.alpha) || !finite_bits(k.beta)) k.brk = 2, k.conv = 1;
      }
      sh.go = !k.conv && !sh.ex.fault;
    }
  }
  __syncthreads();
  return sh.go != 0;
}

// v = (r.z, r.r) of the updated residual; p is visible to every block from here on
template <bool CLUSTER, int T>
__device__ __forceinline__ void pcg_publish(const PcgArgs& a, unsigned int& epoch, const double (&v)[2], int warps,
                                            PcgShared<T>& sh) {
  double total;
  if constexpr (CLUSTER) total = cluster_exchange(epoch, v, warps, sh.ex);
  else total = group_exchange<true>(a.ex, epoch, v, warps, sh.ex);
  if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) sh.last[threadIdx.x >> 5] = total;
}

// Rows of at most three entries (1D grids): the two neighbours' products are added first and the diagonal's last. The
// large terms then meet in one addition, which rounds mirrored rows alike: with a constant coefficient CG
// ends after n / 2 iterations (4,001, 10,000 and 20,000 cells at a tolerance of 1e-12: 2,000, 5,000 and 10,000; one
// sum in the order of the columns takes 3,926, 9,883 and 19,949, whichever form beta has).
template <int CH>
__device__ __forceinline__ double short_row(int w, const double (&v)[CH], const double (&p)[CH]) {
  double s = 0.0;
  if (w > 0) s = v[0] * p[0];
  if (w > 2) s = fma(v[2], p[2], s);
  if (w > 1) s += __dmul_rn(v[1], p[1]);
  return s;
}

// sum of a row's products, entries t of the lane's row at v[32 t], c[32 t]; w is warp-uniform. All loads of
// CH entries are issued before their FMAs. One accumulator: with 16 or more warps on the SM each
// warp's turn at the FP64 pipe comes after the FMA's latency, and a second one would cost an add.
template <bool SHORT, int CH, class LoadV, class LoadC>
__device__ __forceinline__ double pcg_row(int w, const double* p, LoadV v, LoadC c) {
  double s = 0.0;
#pragma unroll 1
  for (int t0 = 0; t0 < w; t0 += CH) {
    double vv[CH], pv[CH];
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      vv[j] = pv[j] = 0.0;
      if (t0 + j < w) {
        vv[j] = v(t0 + j);
        pv[j] = p[c(t0 + j)];
      }
    }
    if (SHORT) s = short_row(w, vv, pv);
    else fma_chain<0>(w - t0, vv, pv, s);
  }
  return s;
}

__device__ __forceinline__ unsigned long long matrix_policy(float keep) {
  unsigned long long pol;
  if (keep >= 1.f) asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
  else if (keep <= 0.f) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  else asm volatile("createpolicy.fractional.L2::evict_normal.L2::evict_first.b64 %0, %1;" : "=l"(pol) : "f"(keep));
  return pol;
}
__device__ __forceinline__ double ld_matrix(const double* a, unsigned long long pol) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ int ld_matrix(const short* a, unsigned long long pol) {
  short v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.s16 %0, [%1], %2;" : "=h"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ int ld_matrix(const int* a, unsigned long long pol) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(pol));
  return v;
}

// The resident form: one block of RT threads per SM, a contiguous range of slices per block, R slices per
// warp, everything a row needs in registers. Two warps per scheduler keep the FP64 pipe busy (a dependent
// FMA can issue as soon as the pipe is free), and each warp more would add its 32 values to every block sum.
// CLUSTER: the grid is one cluster of at most 16 blocks, and the sums go through their shared memory.
constexpr int RT = 256;
constexpr int RMAX = 16;
constexpr int kClusterSlices = 160;
static_assert(kClusterSlices <= 2 * 16 * RT / 32, "two slices per warp");

template <int R, bool CLUSTER>
__global__ void __launch_bounds__(RT, 1) k_pcg_resident(const __grid_constant__ PcgArgs a) {
  __shared__ PcgShared<RT> sh;
  __shared__ int s_off[RT / 32 * R + 1];
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  double* const mv = reinterpret_cast<double*>(pcg_smem);
  int* const mc = reinterpret_cast<int*>(mv + a.cap);
  constexpr int CH = R <= 8 ? 16 : 9;  // entries in flight per row, as the registers allow
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (entry_flag(&a.st->converged)) return;
  const int s0 = a.first[blockIdx.x], ns = a.first[blockIdx.x + 1] - s0;
  const int warps = min(ns, RT / 32);  // that have rows
  if (threadIdx.x == 0) {
    sh.ex.fault = 0;
    sh.k.load(a.st);
  }
  // shared-memory offsets of the block's slices, in order (one warp scans)
  for (int k = threadIdx.x; k < RT / 32 * R; k += RT) s_off[k + 1] = k < ns ? a.width[s0 + k] * 32 : 0;
  if (threadIdx.x == 0) s_off[0] = 0;
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int k0 = 0; k0 < RT / 32 * R; k0 += 32) {
      int e = k0 + lane < RT / 32 * R ? s_off[k0 + lane + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, e, o);
        if (lane >= o) e += up;
      }
      e += run;
      if (k0 + lane < RT / 32 * R) s_off[k0 + lane + 1] = e;
      run = __shfl_sync(0xffffffffu, e, 31);
    }
  }
  __syncthreads();
  const unsigned long long pol = matrix_policy(a.keep);
  // (no block writes to the shared memory of one that has not started)
  if (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  double x[R], r[R], p[R], d[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int ls = warp + RT / 32 * k;
    const int row = (s0 + ls) * 32 + lane;
    const bool in = ls < ns && row < a.n;
    x[k] = in ? a.x[row] : 0.0;
    r[k] = in ? a.r[row] : 0.0;
    p[k] = in ? a.p[row] : 0.0;
    d[k] = in ? __ldg(a.dinv + row) : 0.0;
    if (ls < ns && s_off[ls + 1] <= a.cap) {
      const int off = s_off[ls] + lane, w = (s_off[ls + 1] - s_off[ls]) >> 5, src = __ldg(&a.meta[s0 + ls].x) + lane;
      for (int t = 0; t < w; ++t) {
        mv[off + 32 * t] = __ldg(a.val + src + 32 * t);
        mc[off + 32 * t] = __ldg(a.col + src + 32 * t);
      }
    }
  }
  unsigned int epoch = 0;
  while (true) {
    double q[R];
    double v3[3] = {0.0, 0.0, 0.0};
    auto product = [&](auto short_rows) {
      constexpr bool SHORT = decltype(short_rows)::value;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int ls = warp + RT / 32 * i;
        const int off = s_off[ls], w = (s_off[ls + 1] - off) >> 5;
        q[i] = 0.0;
        if (s_off[ls + 1] <= a.cap) {
          const double* sv = mv + off + lane;
          const int* sc = mc + off + lane;
          q[i] = pcg_row<SHORT, CH>(w, a.p, [&](int t) { return sv[32 * t]; }, [&](int t) { return sc[32 * t]; });
        } else if (ls < ns) {  // (behind the last block's slices the table ends)
          const int src = __ldg(&a.meta[s0 + ls].x) + lane;
          const double* gv = a.val + src;
          const int* gc = a.col + src;
          q[i] = pcg_row<SHORT, CH>(w, a.p, [&](int t) { return ld_matrix(gv + 32 * t, pol); },
                                    [&](int t) { return ld_matrix(gc + 32 * t, pol); });
        }
      }
    };
    if (a.short_rows) product(std::true_type());
    else product(std::false_type());
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (warp + RT / 32 * i < ns) {  // warp-uniform
        const double dq = d[i] * q[i];
        v3[0] = fma(p[i], q[i], v3[0]);
        v3[1] = fma(r[i], dq, v3[1]);
        v3[2] = fma(q[i], dq, v3[2]);
      }
    if (!pcg_step<CLUSTER>(a, epoch, v3, warps, sh)) break;
    const double alpha = sh.k.alpha, beta = sh.k.beta;
    double v[2] = {0.0, 0.0};
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int ls = warp + RT / 32 * i;
      if (ls < ns) {
        const int row = (s0 + ls) * 32 + lane;
        x[i] = fma(alpha, p[i], x[i]);
        r[i] = fma(-alpha, q[i], r[i]);
        const double z = d[i] * r[i];
        p[i] = fma(beta, p[i], z);
        if (row < a.n) a.p[row] = p[i];
        v[0] = fma(r[i], z, v[0]);
        v[1] = fma(r[i], r[i], v[1]);
      }
    }
    pcg_publish<CLUSTER>(a, epoch, v, warps, sh);
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int ls = warp + RT / 32 * i;
    const int row = (s0 + ls) * 32 + lane;
    if (ls < ns && row < a.n) a.x[row] = x[i];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sh.k.store(a.st);
}

// The streaming form, for systems whose rows do not fit the registers of the grid: the same iteration with the
// vectors in memory (each block the same contiguous rows in both passes).
// SPLIT: slices of long rows in units of at most kUnit entries per row, each summed by any warp into shared memory, so
// that a few dozen slices of 125 entries are neither 14 gathers in a row for one warp nor uneven shares
// for the others (28^3 Q2 cubes: 69 us an iteration by slices, 52 by units, 48 with the
// gathers ahead).
constexpr int PT = 1024;  // threads per block (one block per SM)
constexpr int kUnit = 36;

__host__ __device__ constexpr int pcg_units(int width) { return width <= kUnit ? 1 : (width + kUnit - 1) / kUnit; }

// The sums of a warp's segments (entries t < w of the lane's row at src + 32 t, columns counted from `row`, 0 unless they
// are 16-bit differences; next(src, w, row) gives them one after the other): begin() where a segment starts, done(sum) where it ends. Groups of nine entries in three
// buffers: the entries are loaded three steps of three before their products and the vector is gathered one step
// before, across the ends of segments, so that neither latency is waited for.
template <class Col, bool SHORT, class Next, class Begin, class Done>
__device__ __forceinline__ void pcg_segments(const PcgArgs& a, unsigned long long pol, Next next, Begin begin, Done done) {
  const int lane = threadIdx.x & 31;
  int src, w, row, nsrc = 0, nw = 0, nrow = 0;
  if (!next(src, w, row)) return;
  bool more = next(nsrc, nw, nrow);
  double v[3][3], g[3][3];
  int c[3][3];
  auto load = [&](int j, int base, int left) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const bool in = 3 * j + i < left;  // warp-uniform
      v[j][i] = in ? ld_matrix(a.val + base + lane + 32 * (3 * j + i), pol) : 0.0;
      c[j][i] = in ? ld_matrix(reinterpret_cast<const Col*>(a.col) + base + lane + 32 * (3 * j + i), pol) : 0;
    }
  };
  auto gather = [&](int j, int from) {
#pragma unroll
    for (int i = 0; i < 3; ++i) g[j][i] = a.p[from + c[j][i]];
  };
#pragma unroll
  for (int j = 0; j < 3; ++j) load(j, src, w);
  gather(0, row);
  begin();
  double s = 0.0;
  for (int t = 0;;) {
    const bool last = t + 9 >= w;
    const int base = last ? nsrc : src + 32 * (t + 9), left = last ? (more ? nw : 0) : w - t - 9;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      gather((j + 1) % 3, j == 2 && last ? nrow : row);
      if (SHORT && j == 0) s = short_row(w, v[0], g[0]);
      else fma_chain<0>(w - t - 3 * j, v[j], g[j], s);
      load(j, base, left);
    }
    if (last) {
      done(s);
      if (!more) break;
      src = nsrc;
      w = nw;
      row = nrow;
      t = 0;
      s = 0.0;
      more = next(nsrc, nw, nrow);
      begin();
    } else {
      t += 9;
    }
  }
}

template <bool SPLIT, class Col>
__global__ void __launch_bounds__(PT, 1) k_pcg_stream(const __grid_constant__ PcgArgs a) {
  __shared__ PcgShared<PT> sh;
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  double* const part = reinterpret_cast<double*>(pcg_smem);          // [unit][lane]
  int2* const unit = reinterpret_cast<int2*>(part + 32 * a.units);   // first entry, entries per row
  int* const begin = reinterpret_cast<int*>(unit + a.units);         // first unit of the block's slices
  if (entry_flag(&a.st->converged)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = a.first[blockIdx.x], s1 = a.first[blockIdx.x + 1];
  const int row1 = min(a.n, s1 * 32);
  double* const q = !SPLIT && a.qshared ? reinterpret_cast<double*>(pcg_smem) : a.q + 32LL * s0;  // of row 32 s0 on
  const unsigned long long pol = matrix_policy(a.keep);
  if (threadIdx.x == 0) {
    sh.ex.fault = 0;
    sh.k.load(a.st);
  }
  if (SPLIT) {
    for (int k = threadIdx.x; k < s1 - s0; k += PT) begin[k + 1] = pcg_units(a.width[s0 + k]);
    __syncthreads();
    if (threadIdx.x == 0) {
      begin[0] = 0;
      for (int k = 0; k < s1 - s0; ++k) begin[k + 1] += begin[k];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < s1 - s0; k += PT) {
      const int w = a.width[s0 + k], n = pcg_units(w), each = (w + n - 1) / n, src = a.meta[s0 + k].x;
      for (int u = 0; u < n; ++u) unit[begin[k] + u] = make_int2(src + 32 * each * u, min(each, w - each * u));
    }
    __syncthreads();
  }
  unsigned int epoch = 0;
  while (true) {
    double v3[3] = {0.0, 0.0, 0.0};
    if (SPLIT) {
      int u = warp, out = warp;
      pcg_segments<Col, false>(
          a, pol,
          [&](int& src, int& w, int& row) {
            row = 0;
            if (u >= begin[s1 - s0]) return false;
            src = unit[u].x;
            w = unit[u].y;
            u += PT / 32;
            return true;
          },
          [] {},
          [&](double s) {
            part[32 * out + lane] = s;
            out += PT / 32;
          });
      __syncthreads();
    }
    // q of the slice's rows and their share of the sums
    double pr = 0.0, rr = 0.0, dr = 0.0;
    int slice = s0 + warp;
    auto begin_row = [&] {
      const int row = slice * 32 + lane;
      const bool in = row < a.n;
      pr = in ? a.p[row] : 0.0;
      rr = in ? a.r[row] : 0.0;
      dr = in ? __ldg(a.dinv + row) : 0.0;
    };
    auto end_row = [&](double s) {
      const int row = slice * 32 + lane;
      if (row < a.n) q[row - 32 * s0] = s;
      const double ds = dr * s;
      v3[0] = fma(pr, s, v3[0]);
      v3[1] = fma(rr, ds, v3[1]);
      v3[2] = fma(s, ds, v3[2]);
      slice += PT / 32;
    };
    if (SPLIT) {
      while (slice < s1) {
        begin_row();
        const int u1 = begin[slice - s0 + 1];
        int u = begin[slice - s0];
        double s = part[32 * u + lane];
        for (++u; u < u1; ++u) s += part[32 * u + lane];
        end_row(s);
      }
    } else {
      int ahead = slice;
      auto next = [&](int& src, int& w, int& row) {
        if (ahead >= s1) return false;
        row = sizeof(Col) == 2 ? min(ahead * 32 + lane, a.n - 1) : 0;  // (in bounds where there is no row)
        src = __ldg(&a.meta[ahead].x);
        w = __ldg(a.width + ahead);
        ahead += PT / 32;
        return true;
      };
      if (a.short_rows) pcg_segments<Col, true>(a, pol, next, begin_row, end_row);
      else pcg_segments<Col, false>(a, pol, next, begin_row, end_row);
    }
    if (!pcg_step<false>(a, epoch, v3, PT / 32, sh)) break;
    const double alpha = sh.k.alpha, beta = sh.k.beta;
    double v[2] = {0.0, 0.0};
    // (two rows per thread and pass, all their loads issued before the first store)
    for (int i0 = s0 * 32 + threadIdx.x; i0 < row1; i0 += 2 * PT) {
      double pv[2], qv[2], xv[2], rv[2], dv[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = i0 + u * PT;
        const bool in = i < row1;
        pv[u] = in ? a.p[i] : 0.0;
        qv[u] = in ? q[i - 32 * s0] : 0.0;
        xv[u] = in ? a.x[i] : 0.0;
        rv[u] = in ? a.r[i] : 0.0;
        dv[u] = in ? __ldg(a.dinv + i) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = i0 + u * PT;
        if (i < row1) {
          a.x[i] = fma(alpha, pv[u], xv[u]);
          const double ri = fma(-alpha, qv[u], rv[u]);
          const double zi = dv[u] * ri;
          a.r[i] = ri;
          a.p[i] = fma(beta, pv[u], zi);
          v[0] = fma(ri, zi, v[0]);
          v[1] = fma(ri, ri, v[1]);
        }
      }
    }
    pcg_publish<false>(a, epoch, v, PT / 32, sh);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) sh.k.store(a.st);
}

// Rows of at most 32 entries (the SELL-32 SpMV's limit). Per iteration, before (three counter barriers, shuffle
// reductions, scalars in every thread) and now, as slopes between two iteration counts: 4,225 rows of Q1 squares
// 25.5 and 5.3 us on a cluster, 5.5 on the grid; 68,921 of an unstructured tetrahedral mesh 31.2 and 10.0;
// 98,304 of SWIPDG 26.0 and 10.2; 155,480 of P1 tetrahedra 29.7 and 12.2; 2,146,689 of 128^3 Q1 (streaming,
// 727.7 MB of matrix) 209 and 152, 156 with the setup of a solve. The graph form takes 51.7 us for
// 393,216 rows of SWIPDG (27 here) and 264 us for 128^3: AUTO takes this form wherever it applies.
// Longer rows too where the form is left to the library (28^3 Q2 cubes, 185,193 rows of up to 125 entries: 60 us in
// the graph form, 42 here; 15,625 rows 37 and 13); a caller who asks for the persistent form gets it for rows of at most 32.
bool persistent_applies(gdt_context ctx, gdt_matrix m) {
  if (ctx->timing || ctx->solver_launch == GDT_SOLVER_LAUNCH_GRAPH) return false;
  return m->max_row >= 1 && m->rows >= 1 &&
         (m->max_row <= 32 ||
          (ctx->solver_launch == GDT_SOLVER_LAUNCH_AUTO && m->max_row <= 512 && !m->sell_padded));
}

// The slices of every block: equally many, unless rows of different lengths are numbered one kind after the other
// (Q2: vertices, edges, faces, cells), where that leaves blocks with twice the average work; then equal
// shares of entries + 10 per row (the vector operations). Returns the most slices of a block.
int pcg_partition(gdt_matrix m, int blocks, bool by_work, int* first) {
  const int n = int(m->sell_off.size()) - 1;
  const auto work = [&](int s) { return m->sell_off[s] + 320LL * s; };
  long long most = 0;
  for (int b = 0; b <= blocks; ++b) {
    first[b] = int((long long)n * b / blocks);
    if (b > 0) most = std::max(most, work(first[b]) - work(first[b - 1]));
  }
  if (by_work && 10 * most * blocks > 12 * work(n))
    for (int b = 1; b < blocks; ++b) {
      int lo = first[b - 1], hi = n;  // the first slice with at least b shares before it
      while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (work(mid) * blocks < work(n) * b) lo = mid + 1;
        else hi = mid;
      }
      first[b] = lo;
    }
  int slices = 0;
  for (int b = 0; b < blocks; ++b) slices = std::max(slices, first[b + 1] - first[b]);
  return slices;
}

// Runs the iterations after residual_init; fin receives the final state. Returns GDT_EUNSUPPORTED, before anything ran,
// where no cooperative launch of the kernel can be made (the caller then runs the graph form).
gdt_status pcg_persistent(gdt_context ctx, gdt_matrix m, double* x, double* r, double* p, double* q,
                          const double* dinv, KState* st, KState* fin, cudaStream_t s, bool clusters = true) {
  int dev = 0, coop = 0, per_sm = 0;
  long long room = 0;
  GDT_TRY_CUDA(ctx, cudaGetDevice(&dev));
  GDT_TRY_CUDA(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop) return GDT_EUNSUPPORTED;  // the caller runs the graph form
  int blocks = std::min(ctx->num_sms, RT);  // one block per SM
  if (ctx->persistent_blocks > 0) blocks = std::min(blocks, ctx->persistent_blocks);
  const int nslices = int((m->rows + 31) / 32);
  // four slices, one per scheduler, before the next block: 4,225 rows in 34 blocks of four warps take 5.6 us
  // an iteration, in 133 blocks of one warp 6.0 us
  blocks = std::max(1, std::min(blocks, (nslices + 3) / 4));
  // Small systems on one cluster, where one can be had and unless the caller has set limits, which are the grid's. Per
  // iteration on the grid and on a cluster: 20 slices of Q1 squares 4.6 and 3.5 us, 133 5.5 and 5.3, 259 5.6 and
  // 6.3; 42 slices of Q1 cubes 6.3 and 4.7, 106 6.4 and 5.6, 215 6.6 and 8.1 (16 SMs' FP64 pipes).
  const bool cluster = clusters && ctx->persistent_blocks == 0 && ctx->persistent_wait_ns == 0 && m->max_row <= 32 &&
                       nslices <= kClusterSlices;
  if (cluster) blocks = std::min(16, std::max(1, nslices / 4));
  // slices per warp of the resident form; where a block has more rows than its registers hold, the
  // streaming form
  GDT_CHECK(ctx, sell_table(ctx, m, s));
  if (m->max_row > 32 && m->sell_len - m->nnz > m->nnz / 2 + 32768) {  // padding is work
    m->sell_padded = true;
    return GDT_EUNSUPPORTED;
  }
  PcgArgs a;
  const int slices = pcg_partition(m, blocks, !cluster, a.first);
  const int per_warp = (slices + RT / 32 - 1) / (RT / 32);
  const void* fn = per_warp <= 1   ? reinterpret_cast<const void*>(&k_pcg_resident<1, false>)
                   : per_warp <= 2 ? reinterpret_cast<const void*>(&k_pcg_resident<2, false>)
                   : per_warp <= 4 ? reinterpret_cast<const void*>(&k_pcg_resident<4, false>)
                   : per_warp <= 8 ? reinterpret_cast<const void*>(&k_pcg_resident<8, false>)
                   : per_warp <= RMAX ? reinterpret_cast<const void*>(&k_pcg_resident<RMAX, false>)
                                      : reinterpret_cast<const void*>(&k_pcg_stream<false, int>);
  if (cluster)
    fn = per_warp <= 1 ? reinterpret_cast<const void*>(&k_pcg_resident<1, true>)
                       : reinterpret_cast<const void*>(&k_pcg_resident<2, true>);
  int threads = per_warp <= RMAX ? RT : PT;
  int cap = 0;
  size_t dyn = 0;
  a.units = 0;
  a.short_rows = m->max_row <= 3;
  // long rows: eight warps cannot hide the latency of what does not stay in shared memory (20^3 Q2 cubes, four slices a
  // warp: 25 us an iteration resident, 33 streaming by slices; 24^3, eight: 48 resident, 38 streaming by units)
  if (m->max_row > 32 && per_warp > 4) {
    fn = reinterpret_cast<const void*>(&k_pcg_stream<false, int>);
    threads = PT;
    int most = 0;
    for (int b = 0; b < blocks; ++b) {
      int units = 0;
      for (int k = a.first[b]; k < a.first[b + 1]; ++k) units += pcg_units((m->sell_off[k + 1] - m->sell_off[k]) / 32);
      most = std::max(most, units);
    }
    GDT_TRY_CUDA(ctx, allow_shared(ctx, reinterpret_cast<const void*>(&k_pcg_stream<true, int>), &room));
    const long long bytes = 264LL * most + 4LL * (slices + 1);
    if (bytes <= room) {  // (with more there are enough slices for every warp)
      fn = reinterpret_cast<const void*>(&k_pcg_stream<true, int>);
      a.units = most;
      dyn = size_t(bytes);
    }
  } else if (per_warp <= RMAX) {
    GDT_TRY_CUDA(ctx, allow_shared(ctx, fn, &room));
    long long want = 0;  // no more than the block with the most entries has: the rest is L1 for the gathers
    for (int b = 0; b < blocks; ++b)
      want = std::max(want, (long long)m->sell_off[a.first[b + 1]] - m->sell_off[a.first[b]]);
    cap = int(std::max(0LL, std::min(want, room / 12 / 32 * 32)));
    dyn = size_t(cap) * 12;
  }
  // streaming by slices: the columns as 16-bit differences where they fit (10 bytes an entry instead of 12), q in shared
  // memory where it fits. 128^3 Q1, with the setup: 165 us an iteration, 160 and 161 with one of them, 156 with both;
  // 91^3 rows, which L2 holds better: 63 and 62.
  const bool narrow = fn == reinterpret_cast<const void*>(&k_pcg_stream<false, int>) && m->sell_band <= 32767;
  if (narrow) fn = reinterpret_cast<const void*>(&k_pcg_stream<false, short>);
  a.qshared = 0;
  if (threads == PT && a.units == 0) {
    GDT_TRY_CUDA(ctx, allow_shared(ctx, fn, &room));
    if (256LL * slices <= room) {
      a.qshared = 1;
      dyn = size_t(256) * slices;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cluster) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = blocks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&per_sm, fn, &cfg) != cudaSuccess || per_sm < 1) {
      cudaGetLastError();
      return pcg_persistent(ctx, m, x, r, p, q, dinv, st, fin, s, false);
    }
  } else {
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    GDT_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, dyn));
  }
  if (per_sm < 1) return GDT_EUNSUPPORTED;
  // The solve's copy of the matrix, from the pool: values, columns, entries per row of the slices. The values are copied
  // at every solve: the caller may have written them through the CSR pointer.
  struct Copy {
    double* val = nullptr;
    cudaStream_t s;
    ~Copy() {
      if (val) cudaFreeAsync(val, s);
    }
  } copy;
  copy.s = s;
  const size_t entries = size_t(std::max(m->sell_len, 32LL));  // (a multiple of 32: every part is aligned)
  const size_t col_bytes = (narrow ? sizeof(short) : sizeof(int)) * entries;
  if (pool_malloc(ctx, &copy.val, sizeof(double) * entries + col_bytes + sizeof(int) * nslices, s) != cudaSuccess) {
    cudaGetLastError();
    return GDT_EUNSUPPORTED;  // no room for it
  }
  int* const col = reinterpret_cast<int*>(copy.val + entries);
  int* const width = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(col) + col_bytes);
  GDT_CHECK(ctx, sell_fill_nonzero(ctx, m, s, col, copy.val, width, narrow));
  a.n = int(m->rows);
  a.meta = reinterpret_cast<const int2*>(m->sell_meta);
  a.width = width;
  a.col = col;
  a.val = copy.val;
  a.dinv = dinv;
  a.x = x;
  a.r = r;
  a.p = p;
  a.q = q;
  a.st = st;
  // packets and fault flag in the upper half of the scratch (kernels of the setup use its start)
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(ctx->scratch + kScratchDoubles / 2);
  const size_t packets = size_t(2 * kSlot) * blocks;  // two buffers
  if (packets + 16 > kScratchDoubles / 2) return fail(ctx, GDT_EUNSUPPORTED, "persistent solver: grid too large");
  a.ex.slots = words + 16;
  a.ex.fault = reinterpret_cast<unsigned int*>(words);
  a.ex.first = 0;
  a.ex.count = blocks;
  a.ex.wait_ns = ctx->persistent_wait_ns > 0 ? (unsigned long long)ctx->persistent_wait_ns : kBarrierNs;
  a.cap = cap;
  {
    // What of the matrix is not in shared memory stays in L2 where it fits beside the vectors (the resident form's p, five
    // of the streaming form) in 62 % of the cache (80 MB here: its two halves hold some lines twice), four
    // fifths of the room where it does not: a larger share evicts itself. 65^3
    // Q1 rows (89 MB, 56 of them streamed): 41.8 us an iteration with every line evict-first, 30.6 kept;
    // 81^3 (172 MB) 79.1, 73.5 with 65 MB kept, 79.3 with 90; 129^3, where the vectors fill L2, 155 and
    // 163 with 64 MB.
    int l2 = 0;
    GDT_TRY_CUDA(ctx, cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
    const double vectors = (threads == PT ? 40.0 : 8.0) * double(m->rows), room = 0.62 * double(l2) - vectors;
    const double streamed = (narrow ? 10.0 : 12.0) * std::max(0.0, double(m->sell_len) - double(cap) * blocks);
    a.keep = streamed <= room ? 1.f : float(std::max(0.0, 0.8 * room / streamed));
  }
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(words, 0, sizeof(unsigned long long) * (packets + 16), s));
  void* args[] = {&a};
  const cudaError_t le = cudaLaunchKernelExC(&cfg, fn, args);
  if (le == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs available than the device has
    cudaGetLastError();
    return GDT_EUNSUPPORTED;
  }
  GDT_TRY_CUDA(ctx, le);
  ctx->launches++;
  unsigned int fault = 0;
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fault, a.ex.fault, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(fin, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  if (fault) return fail(ctx, GDT_ECUDA, "persistent solver: a grid barrier wait ran out");
  return GDT_OK;
}

}  // namespace

__global__ void k_fill(int n, double* __restrict__ v, double value) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = value;
}
__global__ void k_probe(int n, double* __restrict__ a, double* __restrict__ b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    a[i] = b[i] = 1.0 + 0.001 * double(i % 997);
}

// Picks the SpMV schedule of the fused FP64 CG iteration by timing each valid schedule inside that
// iteration (SpMV + update + direction on scratch vectors, a few real CG steps on A x = probe), not
// back to back: inside the loop the SpMV starts with the vectors the other two kernels just wrote
// dirty in L2, and the schedules rank differently there (128^3 Q1: the staged cp.async schedule
// wins in the loop while 4-lane vector CSR wins back to back). Once per matrix; temporary memory of
// 5 n doubles.
gdt_status tune_cg(gdt_context ctx, gdt_matrix m, const Launch& L0, cudaStream_t s) {
  if (m->cg_sched >= 0) return GDT_OK;
  if (m->pinned) {
    m->cg_sched = m->use_sell ? kSellSchedule : m->spmv_sched;
    return GDT_OK;
  }
  const int n = int(m->rows);
  const size_t vb = sizeof(double) * std::max(n, 1);
  double *x = nullptr, *r = nullptr, *p = nullptr, *q = nullptr, *d = nullptr;
  KState* st = nullptr;
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &x, vb, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &r, vb, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &p, vb, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &q, vb, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &d, vb, s));
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &st, sizeof(KState), s));
  const int pair_blocks = std::max(1, std::min(grid_blocks((n + 1) / 2, TH), ctx->num_sms * 8));
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int timing = ctx->timing;
  ctx->timing = 0;
  float best = FLT_MAX;
  int best_sched = m->spmv_sched;
  const bool sell = sell_prepare(ctx, m, s, true) == GDT_OK;
  for (int sched = 0; sched <= kSellSchedule; ++sched) {
    if (sched < kSchedules ? !schedule_valid(sched, m->max_row) : !sell) continue;
    Launch L = L0;
    L.sched = sched < kSchedules ? sched : L0.sched;
    KState init{};
    init.rho = 1.0;
    init.rr0 = 1.0;
    init.max_iter = 1 << 30;
    cudaMemcpyAsync(st, &init, sizeof(KState), cudaMemcpyHostToDevice, s);
    k_fill<<<L.vec_blocks, TH, 0, s>>>(n, x, 0.0);
    k_fill<<<L.vec_blocks, TH, 0, s>>>(n, d, 1.0);
    k_probe<<<L.vec_blocks, TH, 0, s>>>(n, r, p);
    float total = 0.f;
    bool ok = true;
    for (int it = 0; it < 5; ++it) {
      cudaEventRecord(e0, s);
      if (sched == kSellSchedule) spmv_cg_sell(L, m, p, q, st);
      else spmv_mode<double, 1>(L, m->rp, m->col, m->val, p, q, nullptr, st);
      cudaEventRecord(e1, s);
      k_cg_update_jacobi2<<<pair_blocks, TH, 0, s>>>(n, x, p, r, q, d, st, L.partials, L.ticket);
      k_cg_p_jacobi2<<<pair_blocks, TH, 0, s>>>(n, p, r, d, st);
      if (it >= 2) {
        float ms = 0.f;
        ok = ok && cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess;
        total += ms;
      }
    }
    ok = ok && cudaGetLastError() == cudaSuccess;
    ctx->launches += 18;
    if (ok && total < best) {
      best = total;
      best_sched = sched;
    }
  }
  ctx->timing = timing;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(x, s);
  cudaFreeAsync(r, s);
  cudaFreeAsync(p, s);
  cudaFreeAsync(q, s);
  cudaFreeAsync(d, s);
  cudaFreeAsync(st, s);
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  m->cg_sched = best_sched;
  return GDT_OK;
}

gdt_status solve(gdt_context ctx, gdt_matrix m, const double* b, double* x, const gdt_solver_opts* o,
                 gdt_solve_info* info) {
  cudaStream_t s = ctx->stream;
  cudaStream_t own = nullptr;
  if (s == nullptr) {  // the legacy stream cannot be captured; use a blocking stream ordered with it
    own = ctx->own.exchange(nullptr);  // (a solve of another thread in the meantime makes its own)
    if (!own) GDT_TRY_CUDA(ctx, cudaStreamCreate(&own));
    s = own;
  }
  struct Cleanup {
    gdt_context ctx;
    cudaStream_t st;
    ~Cleanup() {
      if (!st) return;
      cudaStreamSynchronize(st);
      cudaStream_t none = nullptr;
      if (!ctx->own.compare_exchange_strong(none, st)) cudaStreamDestroy(st);
    }
  } cleanup{ctx, own};
  const int n = int(m->rows);
  ctx->last_solver_launch = 0;
  Launch L;
  L.ctx = ctx;
  L.n = n;
  GDT_CHECK(ctx, tune_spmv(ctx, m));
  L.sched = m->spmv_sched;
  L.s = s;
  L.vec_blocks = std::max(1, std::min(grid_blocks(n, TH), ctx->num_sms * 8));
  L.partials = ctx->scratch;
  L.ticket = ctx->counters;
  const int chunk = o->check_every > 0 ? o->check_every : 32;
  const bool mixed = o->precision == GDT_PRECISION_MIXED;
  if (mixed && (o->solver != GDT_SOLVER_CG || o->precond == GDT_PREC_ILU0))
    return fail(ctx, GDT_EUNSUPPORTED, "mixed precision is provided for CG with Jacobi or no preconditioner");
  if (mixed && ctx->solver_launch != GDT_SOLVER_LAUNCH_GRAPH && mixed_mf_applies(m)) {
    // 3D Q1 Laplace matrices: the matrix-free operator, all inner iterations in persistent launches
    const gdt_status ms = solve_mixed_mf(ctx, m, b, x, o, info, s);
    if (ms != GDT_EUNSUPPORTED) {
      ctx->last_solver_launch = GDT_SOLVER_LAUNCH_PERSISTENT;
      return ms;
    }
  }
  if (mixed && ctx->solver_launch != GDT_SOLVER_LAUNCH_GRAPH && !ctx->timing && mixed_stencil_supported(m)) {
    // the other vertex stencils in one launch where the rows fit the registers of the grid
    const gdt_status ms = solve_mixed_resident(ctx, m, b, x, o, info, s);
    if (ms != GDT_EUNSUPPORTED) {
      ctx->last_solver_launch = GDT_SOLVER_LAUNCH_PERSISTENT;
      return ms;
    }
  }
  if (mixed && mixed_stencil_supported(m)) {
    ctx->last_solver_launch = GDT_SOLVER_LAUNCH_GRAPH;
    return solve_mixed_stencil(ctx, m, b, x, o, info, s);
  }
  KState* st = nullptr;
  GDT_TRY_CUDA(ctx, pool_malloc(ctx, &st, sizeof(KState), s));
  KState init{};
  init.tol2 = o->tol * o->tol;
  init.max_iter = o->max_iter;
  std::vector<void*> allocs;
  allocs.push_back(st);
  auto alloc = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (pool_malloc(ctx, &p, bytes, s) != cudaSuccess) return nullptr;
    allocs.push_back(p);
    return p;
  };
  struct Freer {
    std::vector<void*>* a;
    cudaStream_t s;
    ~Freer() {
      for (void* p : *a) cudaFreeAsync(p, s);
    }
  } freer{&allocs, s};
  gdt_solve_info res{};
  if (!mixed) {
    GDT_TRY_CUDA(ctx, cudaMemcpyAsync(st, &init, sizeof(KState), cudaMemcpyHostToDevice, s));
    const size_t vb = sizeof(double) * std::max(n, 1);
    double* r = (double*)alloc(vb);
    double* p = (double*)alloc(vb);
    double* q = (double*)alloc(vb);
    double* dinv = nullptr;
    if (!r || !p || !q) return fail(ctx, GDT_ENOMEM, "solver vectors");
    if (o->precond == GDT_PREC_JACOBI) {
      dinv = (double*)alloc(vb);
      if (!dinv) return fail(ctx, GDT_ENOMEM, "solver vectors");
      k_jacobi_diag<double, double><<<L.vec_blocks, TH, 0, s>>>(n, m->rp, m->col, m->val, dinv);
      GDT_CHECK(ctx, check_launch(ctx, "jacobi"));
    }
    Ilu ilu;
    if (o->precond == GDT_PREC_ILU0) {
      GDT_CHECK(ctx, ilu_setup(ctx, m, ilu, s));
      allocs.push_back(ilu.lu);
      allocs.push_back(ilu.diag);
      allocs.push_back(ilu.lorder);
      allocs.push_back(ilu.uorder);
    }
    KState reached{};  // of a persistent launch
    const int chunk_used = (o->precond == GDT_PREC_ILU0) ? std::min(chunk, 2) : chunk;
    const int max_chunks = o->max_iter / chunk_used + 2;
    if (o->solver == GDT_SOLVER_CG) {
      if (o->precond != GDT_PREC_ILU0) {
        // fused Jacobi (or identity) path
        double* one = dinv;
        if (!one) {
          one = (double*)alloc(vb);
          if (!one) return fail(ctx, GDT_ENOMEM, "solver vectors");
          std::vector<double> ones(n, 1.0);
          GDT_TRY_CUDA(ctx, cudaMemcpyAsync(one, ones.data(), vb, cudaMemcpyHostToDevice, s));
          GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
        }
        bool persistent = persistent_applies(ctx, m), resumed = false;
        if (persistent) {
          residual_init<double>(L, m->rp, m->col, m->val, x, b, r, one, p, st);
          const gdt_status ps = pcg_persistent(ctx, m, x, r, p, q, one, st, &reached, s);
          if (ps == GDT_EUNSUPPORTED) persistent = false;  // x untouched: the graph form starts afresh
          else if (ps != GDT_OK) return ps;
          else ctx->last_solver_launch = GDT_SOLVER_LAUNCH_PERSISTENT;
          // coefficients near 1e290, say: the products that beta is formed from leave the range of a double, the
          // quotients of the classical form need not. The graph form goes on from the last iterate.
          resumed = persistent && reached.breakdown == 2;
          if (resumed) persistent = false;
        }
        if (!persistent) {
          ctx->last_solver_launch = GDT_SOLVER_LAUNCH_GRAPH;
          GDT_CHECK(ctx, tune_cg(ctx, m, L, s));
          // the SELL copy is refreshed at every solve (the caller may have written the CSR values)
          const bool cg_sell = m->cg_sched == kSellSchedule && sell_prepare(ctx, m, s, true) == GDT_OK;
          L.sched = m->cg_sched == kSellSchedule ? m->spmv_sched : m->cg_sched;
          residual_init<double>(L, m->rp, m->col, m->val, x, b, r, one, p, st);
          if (resumed) {  // (the tolerance is relative to the first residual)
            GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&st->rr0, &reached.rr0, sizeof(double), cudaMemcpyHostToDevice, s));
            GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&st->iter, &reached.iter, sizeof(int), cudaMemcpyHostToDevice, s));
          }
          // pairs of rows per thread when every vector is 16-byte aligned (the solver's own are; x is
          // the caller's)
          const bool pairs = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
          const int pair_blocks = std::max(1, std::min(grid_blocks((n + 1) / 2, TH), ctx->num_sms * 8));
          GDT_CHECK(ctx, iterate_chunks(ctx, s, &st->converged, chunk_used, max_chunks, [&] {
            if (cg_sell) spmv_cg_sell(L, m, p, q, st);
            else spmv_mode<double, 1>(L, m->rp, m->col, m->val, p, q, nullptr, st);
            timing_begin(ctx, s, GDT_TIMING_CG_UPDATE);
            if (pairs)
              k_cg_update_jacobi2<<<pair_blocks, TH, 0, s>>>(n, x, p, r, q, one, st, L.partials, L.ticket);
            else
              k_cg_update_jacobi<double, double><<<L.vec_blocks, TH, 0, s>>>(n, x, p, r, q, one, st, L.partials,
                                                                             L.ticket);
            timing_end(ctx, s);
            timing_begin(ctx, s, GDT_TIMING_CG_DIRECTION);
            if (pairs)
              k_cg_p_jacobi2<<<pair_blocks, TH, 0, s>>>(n, p, r, one, st);
            else
              k_cg_p_jacobi<double><<<L.vec_blocks, TH, 0, s>>>(n, p, r, one, st);
            timing_end(ctx, s);
            ctx->launches += 2;
          }));
        }
      } else {
        double* z = (double*)alloc(vb);
        if (!z) return fail(ctx, GDT_ENOMEM, "solver vectors");
        residual_init<double>(L, m->rp, m->col, m->val, x, b, r, nullptr, nullptr, st);
        ilu_apply(ctx, m, ilu, r, z, st, s);
        // rho = r.z, p = z
        k_cg_beta<<<L.vec_blocks, TH, 0, s>>>(n, r, z, st, L.partials, L.ticket);
        GDT_TRY_CUDA(ctx, cudaMemcpyAsync(p, z, vb, cudaMemcpyDeviceToDevice, s));
        ctx->launches++;
        GDT_CHECK(ctx, iterate_chunks(ctx, s, &st->converged, chunk_used, max_chunks, [&] {
          spmv_mode<double, 1>(L, m->rp, m->col, m->val, p, q, nullptr, st);
          k_cg_update<<<L.vec_blocks, TH, 0, s>>>(n, x, p, r, q, st, L.partials, L.ticket);
          ilu_apply(ctx, m, ilu, r, z, st, s);
          k_cg_beta<<<L.vec_blocks, TH, 0, s>>>(n, r, z, st, L.partials, L.ticket);
          k_cg_p<<<L.vec_blocks, TH, 0, s>>>(n, p, z, st);
          ctx->launches += 3;
        }));
      }
    } else {
      // BiCGStab with M = Jacobi / ILU0 / identity
      double* rt = (double*)alloc(vb);
      double* v = (double*)alloc(vb);
      double* y = (double*)alloc(vb);
      double* t = (double*)alloc(vb);
      if (!rt || !v || !y || !t) return fail(ctx, GDT_ENOMEM, "solver vectors");
      GDT_TRY_CUDA(ctx, cudaMemsetAsync(v, 0, vb, s));
      GDT_TRY_CUDA(ctx, cudaMemsetAsync(p, 0, vb, s));
      residual_init<double>(L, m->rp, m->col, m->val, x, b, r, nullptr, nullptr, st);
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(rt, r, vb, cudaMemcpyDeviceToDevice, s));
      auto prec = [&](const double* in, double* out) {
        if (o->precond == GDT_PREC_ILU0) ilu_apply(ctx, m, ilu, in, out, st, s);
        else {
          k_scale<double><<<L.vec_blocks, TH, 0, s>>>(n, out, dinv, in, st);
          ctx->launches++;
        }
      };
      GDT_CHECK(ctx, iterate_chunks(ctx, s, &st->converged, chunk_used, max_chunks, [&] {
        k_bicg_rho<<<L.vec_blocks, TH, 0, s>>>(n, rt, r, st, L.partials, L.ticket);
        k_bicg_p<<<L.vec_blocks, TH, 0, s>>>(n, p, r, v, st);
        prec(p, y);
        spmv_mode<double, 2>(L, m->rp, m->col, m->val, y, v, rt, st);
        k_bicg_s<<<L.vec_blocks, TH, 0, s>>>(n, x, y, r, v, st, L.partials, L.ticket);
        prec(r, q);  // q = M^{-1} s
        spmv_mode<double, 3>(L, m->rp, m->col, m->val, q, t, r, st);
        k_bicg_r<<<L.vec_blocks, TH, 0, s>>>(n, x, q, r, t, st, L.partials, L.ticket);
        ctx->launches += 4;
      }));
    }
    KState fin = reached;
    if (ctx->last_solver_launch != GDT_SOLVER_LAUNCH_PERSISTENT) {
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fin, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
      GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    }
    {
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return fail(ctx, GDT_ECUDA, std::string("krylov: ") + cudaGetErrorString(e));
    }
    // report the true FP64 residual of the returned iterate
    residual64(L, m, x, b, r, L.partials + kScratchDoubles - 1);
    double rr_true = 0;
    GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&rr_true, L.partials + kScratchDoubles - 1, sizeof(double),
                                      cudaMemcpyDeviceToHost, s));
    GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    res.iterations = fin.iter;
    res.refinements = 0;
    res.rel_residual = fin.rr0 > 0 ? std::sqrt(rr_true / fin.rr0) : 0.0;
    res.converged = (fin.breakdown == 0) && (fin.rr0 == 0 || fin.rr <= fin.tol2 * fin.rr0);
  } else {
    // ---------------------------------------------------- FP64 iterative refinement, FP32 inner CG
    const size_t vb = sizeof(double) * std::max(n, 1), fb = sizeof(float) * std::max(n, 1);
    double* r = (double*)alloc(vb);
    float* val32 = (float*)alloc(sizeof(float) * (m->nnz + 8));
    float* r32 = (float*)alloc(fb);
    float* d32 = (float*)alloc(fb);
    float* p32 = (float*)alloc(fb);
    float* q32 = (float*)alloc(fb);
    float* dinv32 = (float*)alloc(fb);
    double* scal = (double*)alloc(sizeof(double) * 4);
    if (!r || !val32 || !r32 || !d32 || !p32 || !q32 || !dinv32 || !scal) return fail(ctx, GDT_ENOMEM, "solver vectors");
    k_to_float<<<ctx->num_sms * 8, TH, 0, s>>>(m->nnz, m->val, val32);
    ctx->launches++;
    if (o->precond == GDT_PREC_JACOBI)
      k_jacobi_diag<float, double><<<L.vec_blocks, TH, 0, s>>>(n, m->rp, m->col, m->val, dinv32);
    else {
      std::vector<float> ones(n, 1.0f);
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(dinv32, ones.data(), fb, cudaMemcpyHostToDevice, s));
      GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    }
    ctx->launches++;
    const double inner_tol = o->inner_tol > 0 ? o->inner_tol : 1e-3;
    double rr0 = -1.0, rr = 0.0;
    int total_iter = 0, refinements = 0;
    bool ok = false;
    double* rr_dev = scal;
    for (int outer = 0; outer < 200; ++outer) {
      residual64(L, m, x, b, r, rr_dev);
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&rr, rr_dev, sizeof(double), cudaMemcpyDeviceToHost, s));
      GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
      if (rr0 < 0) rr0 = rr;
      if (!std::isfinite(rr)) break;
      if (rr <= o->tol * o->tol * rr0 || rr == 0.0) {
        ok = true;
        break;
      }
      if (total_iter >= o->max_iter) break;
      // inner: A d = r / ||r|| in FP32, d0 = 0
      k_scale_to_float<<<L.vec_blocks, TH, 0, s>>>(n, r, rr_dev, r32);
      GDT_TRY_CUDA(ctx, cudaMemsetAsync(d32, 0, fb, s));
      KState in = init;
      in.tol2 = inner_tol * inner_tol;
      in.max_iter = std::max(1, o->max_iter - total_iter);
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(st, &in, sizeof(KState), cudaMemcpyHostToDevice, s));
      k_init_from_rhs<float><<<L.vec_blocks, TH, 0, s>>>(n, r32, dinv32, p32, st, L.partials, L.ticket);
      ctx->launches += 2;
      GDT_CHECK(ctx, iterate_chunks(ctx, s, &st->converged, chunk, in.max_iter / chunk + 2, [&] {
        spmv_mode<float, 1>(L, m->rp, m->col, val32, p32, q32, nullptr, st);
        k_cg_update_jacobi<float, float><<<L.vec_blocks, TH, 0, s>>>(n, d32, p32, r32, q32, dinv32, st, L.partials,
                                                                     L.ticket);
        k_cg_p_jacobi<float><<<L.vec_blocks, TH, 0, s>>>(n, p32, r32, dinv32, st);
        ctx->launches += 2;
      }));
      KState fin;
      GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fin, st, sizeof(KState), cudaMemcpyDeviceToHost, s));
      GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
      total_iter += fin.iter;
      k_correct<<<L.vec_blocks, TH, 0, s>>>(n, x, d32, rr_dev);
      ctx->launches++;
      refinements++;
      if (fin.breakdown) break;
    }
    {
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return fail(ctx, GDT_ECUDA, std::string("mixed krylov: ") + cudaGetErrorString(e));
    }
    res.iterations = total_iter;
    res.refinements = refinements;
    res.rel_residual = rr0 > 0 ? std::sqrt(rr / rr0) : 0.0;
    res.converged = ok ? 1 : 0;
  }
  if (info) *info = res;
  if (!res.converged) return fail(ctx, GDT_ENOCONV, "linear solver did not converge");
  return GDT_OK;
}

}  // namespace gdt
