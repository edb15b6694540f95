// The batched solver's main kernel (batch.cu holds the host side and the fixed-size team kernel).
//
// One cooperative launch, one block per SM. The blocks are divided into teams of as many blocks as the host's
// plan gives them; a team takes problems from a list, largest first, and solves each on all of its
// blocks. What bounds a solve is the FP64 pipe (a warp instruction holds a quarter of an SM for 64
// cycles), so that is what is economised:
//  * CG runs on the Jacobi-scaled system (D^-1/2 A D^-1/2, unit diagonal): four (P1) or eight (Q1)
//    multiply-adds a row for the product and no products with D^-1 elsewhere. P1 couples no vertices
//    across a hypotenuse (the gradients are orthogonal), so the seven-entry rows have five nonzeros.
//  * beta is formed with alpha, from sums taken with q = A p (as in the persistent single solver), so
//    x, r and p are updated in one pass.
//  * The stopping test needs |r|^2 = sum d_i r^_i^2 of the unscaled residual; r^.r^ >= |r|^2 / max d gives
//    |r|^2 >= min d (r^.r^), and while that bound is above twice the threshold the sum is not formed.
//  * x, r, q and, for one-block teams, p and the couplings live in shared memory where a block's rows fit.
// The scaled couplings are rounded once more than the assembled ones, which alone would leave the solution
// three to eight times further off where those are exact (kappa constant per quadrant, 512 squares:
// 6e-12 against 1e-12 at a tolerance of 1e-10). So at one and at two thirds of the way to the tolerance
// (in digits) the residual is replaced by that of the assembled rows: what is iterated after that is
// small enough for the rounding not to matter, and there is enough of it to remove what has gathered
// (replaced only 100x before the threshold it stays at 3e-12). It costs sixteen iterations' work.
// A problem with a diagonal entry that is not positive (a coefficient <= 0) keeps the unscaled
// preconditioned iteration. So does one whose tolerance is below what the rounding of the couplings leaves in the
// residual, about n^2 eps where they are alike (kappa constant per quadrant): a replacement puts that back after CG
// has done with the smooth part, which takes more iterations then. At 1e-12 256, 400 and 512 squares took 1,079,
// 1,746 and 2,414 iterations scaled, with errors up to five times as large, and take 1,075, 1,674 and
// 2,146 unscaled; 16 problems of 512 squares 254 and 287 ms, 32 of 256 65 and 80.
#pragma once
#include <type_traits>

#include "exchange.cuh"
#include "structured.cuh"

namespace gdt {

struct TeamPlace {  // of one block
  int first, count;     // its team: blocks first .. first + count - 1
  int list;             // the list its team starts with (0: the larger problems, then 1; 1: only 1)
  int pad;
  long long scratch;    // word offset of the team's scratch
};

struct TeamBatchArgs {
  const TeamPlace* place;
  const int* probs;  // list 0, then list 1
  int count[2];
  int* taken;        // per list, problems taken so far
  const long long* off;
  const long long* eoff;
  const int* cells;
  const double* kappa;
  int kappa_elems;   // 0: kappa[4 i + q] per quadrant; 1: per element from eoff[i]
  double force;
  double tol2;
  int max_iter;
  double* x;
  double* stencil_out;
  int* iters;
  double* relres;
  int* status;
  double* scratch;
  ExchangeView ex;   // slots, fault and wait limit (first and count come from the place)
  int smem_words;    // doubles of dynamic shared memory
  double K[2][4][4];  // local stiffness: P1 triangle types t (3 x 3), or Q1 (K[0], 4 x 4)
};

// threads per block, and rows a thread has in flight in the product and in the update: two warps per scheduler keep
// the FP64 pipe busy, and each warp more adds its 32 values to every block sum (16 problems of 512
// squares: 238 ms; 512 threads with half the rows 261 ms, 1024 267 ms; 4 instead of 8 update rows 267 ms)
constexpr int TB = 256, UA = 4, UB = 8;

// couplings of a row kept once per edge: +x, +y and, for Q1, +x+y and -x+y
template <int NS>
__host__ __device__ constexpr int team_couplings() {
  return NS == 7 ? 2 : 4;
}
// arrays of a problem: p, q, r, x, d, s and the couplings
template <int NS>
__host__ __device__ constexpr int team_arrays() {
  return 6 + team_couplings<NS>();
}
// words of one array of an n x n problem: its rows and a line of zeros on both sides
__host__ __device__ inline long long team_stride(long long n) {
  const long long rows = (n + 1) * (n + 1), pad = (n + 3) / 2 * 2 + 2;
  return (rows + 2 * pad + 31) / 32 * 32;
}
__host__ __device__ inline int team_pad(int n) { return (n + 3) / 2 * 2 + 2; }

// An array that only the owner of a row reads: its first rows in shared memory, from `split` on in scratch.
// A group of rows that starts below the split ends below it.
struct OwnRows {
  double *low, *high;
  int split;
  __device__ __forceinline__ double* at(int i) const { return i < split ? low : high; }
  __device__ __forceinline__ double& operator[](int i) const { return at(i)[i]; }
};

// a problem's arrays, each indexed by the row (p, d, s and the couplings in scratch or shared memory)
template <int NS>
struct TeamArrays {
  double *p, *d, *s;
  OwnRows q, r, x;
  double* c[team_couplings<NS>()];
};

struct TeamScalars {
  double rho, alpha, beta, stop, dmin;
  double mark, step;  // |r|^2 at which the residual is replaced next, and the factor to the mark after that
  int iter, conv, need, go;
  int replace;  // the residual is replaced after this update
};

template <int NS>
struct TeamRow {
  // s + sum of coupling times neighbour; the loads of a row are one struct so that several rows are in flight
  double cp[2 * team_couplings<NS>()], pn[2 * team_couplings<NS>()];
  __device__ __forceinline__ void load(const TeamArrays<NS>& w, int i, int nv) {
    constexpr int C = team_couplings<NS>();
    const int off[4] = {1, nv, nv + 1, nv - 1};
#pragma unroll
    for (int k = 0; k < C; ++k) {
      cp[2 * k] = w.c[k][i];
      pn[2 * k] = w.p[i + off[k]];
      cp[2 * k + 1] = w.c[k][i - off[k]];
      pn[2 * k + 1] = w.p[i - off[k]];
    }
  }
  __device__ __forceinline__ double dot(double s) const {
#pragma unroll
    for (int k = 0; k < 2 * team_couplings<NS>(); ++k) s = fma(cp[k], pn[k], s);
    return s;
  }
  // the whole row in the order of its columns, as batch_kernel adds it (the diagonal first leaves up to three times the
  // error where kappa is constant per quadrant: 256 squares, tolerance 1e-12)
  __device__ __forceinline__ double dot_by_column(double d, double p) const {
    constexpr int C = team_couplings<NS>();
    constexpr int order[8] = {5, 3, 7, 1, 0, 6, 2, 4};
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k == 4) s = fma(d, p, s);
      if (order[k] < 2 * C) s = fma(cp[order[k]], pn[order[k]], s);
    }
    return s;
  }
};

// rows i0 + TB u for u < U, in full groups, then one by one: no FP64 instruction runs masked off
template <int U, class Body>
__device__ __forceinline__ void team_rows(int lo, int hi, Body body) {
  int base = lo;
  for (; base + U * TB <= hi; base += U * TB) body(base + (int)threadIdx.x, std::integral_constant<int, U>());
  for (int i = base + (int)threadIdx.x; i < hi; i += TB) body(i, std::integral_constant<int, 1>());
}

// the assembled row of vertex (ix, iy) with the Dirichlet constraints, by slot of the 3 x 3 neighbourhood; nel
// elements meet there, nbad counts their non-finite kappa
template <int NS>
__device__ __forceinline__ void team_row(const TeamBatchArgs& a, int prob, int n, int ix, int iy, double (&acc)[9],
                                         int& nel, int& nbad) {
  const double* kq = a.kappa + 4LL * prob;
  const double* ke = a.kappa + (a.kappa_elems ? a.eoff[prob] : 0);
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.0;
  nel = 0;
#pragma unroll
  for (int cv = 0; cv < 4; ++cv) {
    const int cx = ix - (cv & 1), cy = iy - ((cv >> 1) & 1);
    if (cx < 0 || cy < 0 || cx >= n || cy >= n) continue;
    const long long cell = cx + (long long)n * cy;
    auto finite = [](double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; };
    if constexpr (NS == 7) {
#pragma unroll
      for (int tt = 0; tt < 2; ++tt)
#pragma unroll
        for (int li = 0; li < 3; ++li) {
          if (local_corner(2, true, tt, li) != cv) continue;
          const double kap = a.kappa_elems ? ke[2 * cell + tt] : kq[(cx >= n / 2 ? 1 : 0) + (cy >= n / 2 ? 2 : 0)];
          nbad += !finite(kap);
          ++nel;
#pragma unroll
          for (int lj = 0; lj < 3; ++lj) acc[slot_between(2, cv, local_corner(2, true, tt, lj))] += kap * a.K[tt][li][lj];
        }
    } else {
      const double kap = a.kappa_elems ? ke[cell] : kq[(cx >= n / 2 ? 1 : 0) + (cy >= n / 2 ? 2 : 0)];
      nbad += !finite(kap);
      ++nel;
#pragma unroll
      for (int lj = 0; lj < 4; ++lj) acc[slot_between(2, cv, lj)] += kap * a.K[0][cv][lj];
    }
  }
  auto on_boundary = [&](int jx, int jy) { return jx == 0 || jy == 0 || jx == n || jy == n; };
  const bool bnd = on_boundary(ix, iy);
#pragma unroll
  for (int sl = 0; sl < 9; ++sl) {
    if (bnd) acc[sl] = sl == 4 ? 1.0 : 0.0;
    else if (on_boundary(ix + sl % 3 - 1, iy + sl / 3 - 1)) acc[sl] = 0.0;
  }
}

// b - A x of row i with the assembled row; x in global memory
template <int NS>
__device__ __forceinline__ double team_residual(const TeamBatchArgs& a, int prob, int n, int i, const double* x,
                                                double b_inner) {
  const int nv = n + 1, ix = i % nv, iy = i / nv;
  if (ix == 0 || iy == 0 || ix == n || iy == n) return 0.0 - x[i];
  double acc[9];
  int nel, nbad = 0;
  team_row<NS>(a, prob, n, ix, iy, acc, nel, nbad);
  double s = 0.0;
#pragma unroll
  for (int sl = 0; sl < 9; ++sl)
    if (NS == 9 || (sl != 0 && sl != 2 && sl != 6 && sl != 8)) s = fma(acc[sl], x[i + (sl % 3 - 1) + (sl / 3 - 1) * nv], s);
  return b_inner - s;
}

// rows of the problem: couplings, diagonal, the exported stencil; the counts of non-finite kappa values and
// loads and of diagonal entries that are not positive, and the smallest diagonal
template <int NS>
__device__ void team_assemble(const TeamBatchArgs& a, int prob, int n, int lo, int hi, const TeamArrays<NS>& w,
                              double& bad, double& nonpos, double& dmin) {
  const int nv = n + 1;
  const double h = 1.0 / n;
  const long long off = a.off[prob];
  int nbad = 0, nneg = 0;
  dmin = INFINITY;
  for (int i = lo + threadIdx.x; i < hi; i += TB) {
    const int ix = i % nv, iy = i / nv;
    double acc[9];
    int nel;
    team_row<NS>(a, prob, n, ix, iy, acc, nel, nbad);
    if (a.stencil_out) {
      constexpr int p1[7] = {0, 1, 3, 4, 5, 7, 8};
#pragma unroll
      for (int k = 0; k < NS; ++k) a.stencil_out[NS * (off + i) + k] = acc[NS == 9 ? k : p1[k]];
    }
    w.c[0][i] = acc[5];
    w.c[1][i] = acc[7];
    if constexpr (NS == 9) {
      w.c[2][i] = acc[8];
      w.c[3][i] = acc[6];
    }
    w.d[i] = acc[4];
    nneg += !(acc[4] > 0.0);
    if (!(ix == 0 || iy == 0 || ix == n || iy == n)) dmin = acc[4] < dmin ? acc[4] : dmin;
    const double per_el = NS == 7 ? 0.5 * h * h / 3.0 : 0.25 * h * h;
    nbad += (__double2hiint(a.force * per_el * nel) & 0x7ff00000) == 0x7ff00000;
  }
  bad = double(nbad);
  nonpos = double(nneg);
}

// One problem on the blocks of the team. Rows are dealt out in contiguous ranges; row i's neighbours in other
// ranges are read from the team's scratch (p and the couplings), everything else only by its owner.
template <int NS, bool SCALED>
__device__ void team_cg(const TeamBatchArgs& a, const ExchangeView& ex, unsigned int& epoch, int prob, int n, int lo,
                        int hi, const TeamArrays<NS>& w, ExchangeShared<TB>& sh, double* total, TeamScalars& k,
                        double b_inner) {
  double* const xout = a.x + a.off[prob];
  const int nv = n + 1;
  constexpr int C = team_couplings<NS>();
  // scale the rows: s = d^-1/2 (d^-1 for the unscaled iteration), couplings times s of both ends
  for (int i = lo + threadIdx.x; i < hi; i += TB) w.s[i] = SCALED ? 1.0 / sqrt(w.d[i]) : 1.0 / w.d[i];
  double none[1] = {0.0};
  if (SCALED) {
    group_exchange<true>(ex, epoch, none, TB / 32, sh);
    const int offs[4] = {1, nv, nv + 1, nv - 1};
    for (int i = lo + threadIdx.x; i < hi; i += TB) {
      const double si = w.s[i];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const double v = w.c[c][i];
        if (v != 0.0) w.c[c][i] = v * si * w.s[i + offs[c]];
      }
    }
  }
  double v2[2] = {0.0, 0.0};
  for (int i = lo + threadIdx.x; i < hi; i += TB) {
    const int ix = i % nv, iy = i / nv;
    const double b = ix == 0 || iy == 0 || ix == n || iy == n ? 0.0 : b_inner;
    const double si = w.s[i], r = SCALED ? si * b : b, z = SCALED ? r : si * r;
    w.x[i] = 0.0;
    w.r[i] = r;
    w.p[i] = z;
    v2[0] = fma(r, z, v2[0]);
    v2[1] = fma(b, b, v2[1]);
  }
  {
    const double t = group_exchange<true>(ex, epoch, v2, TB / 32, sh);
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) total[3 + (threadIdx.x >> 5)] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      k.rho = total[3];
      k.stop = a.tol2 * total[4];
      k.step = cbrt(a.tol2);
      k.mark = SCALED ? k.step * total[4] : -1.0;
      k.iter = 0;
      k.conv = total[4] == 0.0;
      k.need = 0;
      k.replace = 0;
      k.go = !k.conv && !sh.fault;
    }
    __syncthreads();
  }
  bool first = true;
  while (k.go) {
    // q = A p with p.q, z.q, q.M^-1 q
    double v3[3] = {0.0, 0.0, 0.0};
    team_rows<UA>(lo, hi, [&](int i0, auto rows) {
      constexpr int U = decltype(rows)::value;
      double *const wr = w.r.at(i0), *const wq = w.q.at(i0);
      TeamRow<NS> row[U];
      double p[U], r[U], d[U], s[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + TB * u;
        row[u].load(w, i, nv);
        p[u] = w.p[i];
        r[u] = wr[i];
        d[u] = s[u] = 1.0;
        if (!SCALED) {
          d[u] = w.d[i];
          s[u] = w.s[i];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const double q = SCALED ? row[u].dot(p[u]) : row[u].dot_by_column(d[u], p[u]);
        const double mq = SCALED ? q : s[u] * q;
        wq[i0 + TB * u] = q;
        v3[0] = fma(p[u], q, v3[0]);
        v3[1] = fma(r[u], mq, v3[1]);
        v3[2] = fma(q, mq, v3[2]);
      }
    });
    {
      const double t = group_exchange<false>(ex, epoch, v3, TB / 32, sh);
      if (threadIdx.x < 96) {
        const double inv = threadIdx.x == 0 ? 1.0 / t : 0.0;
        if ((threadIdx.x & 31) == 0) total[threadIdx.x >> 5] = t;
        asm volatile("bar.sync 1, 96;" ::: "memory");
        if (threadIdx.x == 0) {
          int stopped = 0;
          if (!first) {  // the iteration before: its sums were formed beside this product
            k.rho = total[3];
            k.iter += 1;
            if (k.need && total[4] <= k.stop) k.conv = stopped = 1;
            if (k.iter >= a.max_iter) stopped = 1;
          }
          if (!stopped && !(t > 0.0)) {  // breakdown: not SPD, or the exact solution reached
            k.conv = t == 0.0;
            stopped = 1;
          }
          if (!stopped) {
            k.alpha = k.rho * inv;
            k.beta = fma(k.alpha * inv, total[2], fma(-2.0 * inv, total[1], 1.0));
            const double least = 0.5 * k.dmin * (k.beta * k.rho);  // of |r|^2 after this update
            k.need = !SCALED || !(least > k.stop);
            k.replace = !(least > k.mark);  // at |r| = tol^(1/3) |b| and tol^(2/3) |b|
            if (k.replace) k.mark *= k.mark * k.step > 2.0 * k.stop ? k.step : -1.0;
          }
          k.go = !stopped && !sh.fault;
        }
      }
      __syncthreads();
      first = false;
      if (!k.go) break;
    }
    const double alpha = k.alpha, beta = k.beta;
    const int need = k.need;
    double v[2] = {0.0, 0.0};
    team_rows<UB>(lo, hi, [&](int i0, auto rows) {
      constexpr int U = decltype(rows)::value;
      double *const wr = w.r.at(i0), *const wq = w.q.at(i0), *const wx = w.x.at(i0);
      double p[U], q[U], x[U], r[U], s[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + TB * u;
        p[u] = w.p[i];
        q[u] = wq[i];
        x[u] = wx[i];
        r[u] = wr[i];
        s[u] = SCALED ? 1.0 : w.s[i];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + TB * u;
        r[u] = fma(-alpha, q[u], r[u]);
        const double z = SCALED ? r[u] : s[u] * r[u];
        wx[i] = fma(alpha, p[u], x[u]);
        wr[i] = r[u];
        w.p[i] = fma(beta, p[u], z);
        v[0] = fma(r[u], z, v[0]);
      }
      if (need) {
#pragma unroll
        for (int u = 0; u < U; ++u) v[1] = fma(SCALED ? w.d[i0 + TB * u] * r[u] : r[u], r[u], v[1]);
      }
    });
    if (SCALED && k.replace) {
      // r = b - A x from the assembled rows; p keeps its conjugate part
      for (int i = lo + threadIdx.x; i < hi; i += TB) xout[i] = w.s[i] * w.x[i];
      group_exchange<true>(ex, epoch, none, TB / 32, sh);
      v[0] = v[1] = 0.0;
      for (int i = lo + threadIdx.x; i < hi; i += TB) {
        const double res = team_residual<NS>(a, prob, n, i, xout, b_inner), r = w.s[i] * res;
        w.p[i] += r - w.r[i];
        w.r[i] = r;
        v[0] = fma(r, r, v[0]);
        v[1] = fma(res, res, v[1]);
      }
    }
    const double t = group_exchange<true>(ex, epoch, v, TB / 32, sh);
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) total[3 + (threadIdx.x >> 5)] = t;
  }
  __syncthreads();
}

template <int NS>
__device__ void team_solve(const TeamBatchArgs& a, const ExchangeView& ex, unsigned int& epoch, int prob,
                           double* scratch, double* smem, ExchangeShared<TB>& sh, double* total, TeamScalars& k) {
  const int n = a.cells[prob];
  const int nv = n + 1;
  const int N = nv * nv;
  const int rank = blockIdx.x - ex.first;
  const int lo = int((long long)N * rank / ex.count), hi = int((long long)N * (rank + 1) / ex.count);
  const long long stride = team_stride(n);
  const int pad = team_pad(n);
  constexpr int C = team_couplings<NS>();
  TeamArrays<NS> w;
  w.p = scratch + pad;
  w.d = w.p + stride;
  w.s = w.d + stride;
#pragma unroll
  for (int c = 0; c < C; ++c) w.c[c] = w.s + (c + 1) * stride;
  // arrays only their owner reads move to shared memory, in the order of their accesses per iteration
  // (r three, q and x two); the one that no longer fits with its first rows
  int room = a.smem_words;
  double* sm = smem;
  auto own = [&](OwnRows& rows, int k) {
    rows.high = w.s + (C + k) * stride;
    const int take = hi - lo <= room ? hi - lo : room / (UB * TB) * (UB * TB);
    rows.low = sm - lo;
    rows.split = lo + take;
    sm += take;
    room -= take;
  };
  own(w.r, 1);
  own(w.q, 2);
  own(w.x, 3);
  if (ex.count == 1) {  // with no other block to read them, the padded ones too
    auto padded = [&](double*& ptr) {
      if (N + 2 * pad <= room) {
        ptr = sm + pad;
        sm += N + 2 * pad;
        room -= N + 2 * pad;
      }
    };
    padded(w.p);
#pragma unroll
    for (int c = 0; c < C; ++c) padded(w.c[c]);
  }
  // zeros around the arrays that are read across a row's neighbours
  auto clear_pads = [&](double* ptr) {
    if (rank == 0)
      for (int i = threadIdx.x; i < pad; i += TB) ptr[i - pad] = 0.0;
    if (rank == ex.count - 1)
      for (int i = threadIdx.x; i < pad; i += TB) ptr[N + i] = 0.0;
  };
  clear_pads(w.p);
#pragma unroll
  for (int c = 0; c < C; ++c) clear_pads(w.c[c]);
  double v3[3], dmin;
  team_assemble<NS>(a, prob, n, lo, hi, w, v3[0], v3[1], dmin);
  // the smallest diagonal of the block travels with the counts, as a third value that only thread 0 holds
  for (int o = 16; o > 0; o >>= 1) dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
  if ((threadIdx.x & 31) == 0) sh.part[0][threadIdx.x >> 5] = dmin;
  __syncthreads();
  v3[2] = 0.0;
  if (threadIdx.x == 0) {
    v3[2] = sh.part[0][0];
    for (int t = 1; t < TB / 32; ++t) v3[2] = fmin(v3[2], sh.part[0][t]);
  }
  __syncthreads();
  {
    const double t = group_exchange<true>(ex, epoch, v3, TB / 32, sh);
    if (threadIdx.x < 96 && (threadIdx.x & 31) == 0) total[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = ex.count == 1 ? total[2] : sh.packet[2][0];
      for (int t2 = 1; t2 < ex.count; ++t2) m = sh.packet[2][t2] < m ? sh.packet[2][t2] : m;
      k.dmin = m;
    }
    __syncthreads();
  }
  const double bad = total[0], nonpos = total[1];
  const double h = 1.0 / n;
  const double b_inner = a.force * (NS == 7 ? 0.5 * h * h / 3.0 : 0.25 * h * h) * (NS == 7 ? 6 : 4);
  double* x = a.x + a.off[prob];
  int st = GDT_ENAN;
  double relres = 0.0;
  __syncthreads();
  if (bad > 0.0 || sh.fault) {  // skipped: x = 0
    for (int i = lo + threadIdx.x; i < hi; i += TB) x[i] = 0.0;
    if (threadIdx.x == 0) k.iter = k.conv = 0;
    __syncthreads();
  } else {
    const double rounding = 2.5 * 1.1102230246251565e-16 * n * n;  // 7.3e-11 for 512 squares
    const bool scaled = nonpos == 0.0 && a.tol2 >= rounding * rounding;
    // the scaled system with d^1/4 times the load (a power of two: the same bits): its sums go with b^2 / d and with
    // b^2, and both stay in the range of a double for any coefficient
    const int e = scaled && isfinite(k.dmin) ? ilogb(k.dmin) / 4 : 0;
    const double unit = scalbn(1.0, -e);
    if (scaled) team_cg<NS, true>(a, ex, epoch, prob, n, lo, hi, w, sh, total, k, scalbn(b_inner, e));
    else team_cg<NS, false>(a, ex, epoch, prob, n, lo, hi, w, sh, total, k, b_inner);
    // the solution and its true relative residual
    for (int i = lo + threadIdx.x; i < hi; i += TB) x[i] = scaled ? w.s[i] * w.x[i] * unit : w.x[i];
    double v[2] = {0.0, 0.0};
    double none[1] = {0.0};
    group_exchange<true>(ex, epoch, none, TB / 32, sh);
    for (int i = lo + threadIdx.x; i < hi; i += TB) {
      const int ix = i % nv, iy = i / nv;
      const double b = ix == 0 || iy == 0 || ix == n || iy == n ? 0.0 : b_inner;
      const double res = team_residual<NS>(a, prob, n, i, x, b_inner);
      v[0] = fma(res, res, v[0]);
      v[1] = fma(b, b, v[1]);
    }
    const double t = group_exchange<true>(ex, epoch, v, TB / 32, sh);
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) total[threadIdx.x >> 5] = t;
    __syncthreads();
    relres = total[1] > 0.0 ? sqrt(total[0] / total[1]) : 0.0;
    st = sh.fault ? GDT_ETIMEOUT : k.conv ? GDT_OK : GDT_ENOCONV;
  }
  if (rank == 0 && threadIdx.x == 0) {
    a.iters[prob] = k.conv ? k.iter : -k.iter - 1;
    a.relres[prob] = relres;
    a.status[prob] = sh.fault ? GDT_ETIMEOUT : st;
  }
  __syncthreads();
}

template <int NS>
__global__ void __launch_bounds__(TB, 1) batch_team_kernel(const __grid_constant__ TeamBatchArgs a) {
  extern __shared__ __align__(16) double team_smem[];
  __shared__ ExchangeShared<TB> sh;
  __shared__ double total[5];
  __shared__ TeamScalars k;
  const TeamPlace place = a.place[blockIdx.x];
  ExchangeView ex = a.ex;
  ex.first = place.first;
  ex.count = place.count;
  if (threadIdx.x == 0) sh.fault = 0;
  unsigned int epoch = 0;
  int list = place.list, mine = 0;
  for (;;) {
    // the team's first block takes the next problem; the others learn it by the exchange (as a sum)
    double v[1] = {0.0};
    if (blockIdx.x == ex.first && threadIdx.x == 0) v[0] = double(mine = atomicAdd(a.taken + list, 1));
    const double t = group_exchange<true>(ex, epoch, v, TB / 32, sh);
    if (threadIdx.x == 0) total[0] = t;
    __syncthreads();
    const int it = int(total[0]);
    const bool lost = sh.fault != 0;  // a wait ran out: what is left of the lists is reported, not solved
    __syncthreads();
    if (lost) break;
    if (it >= a.count[list]) {
      if (++list < 2) continue;
      break;
    }
    team_solve<NS>(a, ex, epoch, a.probs[(list ? a.count[0] : 0) + it], a.scratch + place.scratch, team_smem, sh, total, k);
  }
  if (sh.fault && blockIdx.x == ex.first && threadIdx.x == 0)
    for (; list < 2; mine = ++list < 2 ? atomicAdd(a.taken + list, 1) : 0)
      for (int it = mine; it < a.count[list]; it = atomicAdd(a.taken + list, 1)) {
        const int prob = a.probs[(list ? a.count[0] : 0) + it];
        a.iters[prob] = -1;
        a.relres[prob] = 0.0;
        a.status[prob] = GDT_ETIMEOUT;
      }
}

}  // namespace gdt
