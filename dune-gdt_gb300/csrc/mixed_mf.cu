// Mixed-precision CG for 3D Q1 Laplace matrices with element coefficients (the solve behind
// ConstMatrixOperator::apply_inverse, operators/matrix-based.hh:131-159, for the matrices of
// LocalLaplaceIntegrand on cube grids): FP32 inner iterations in the Chronopoulos-Gear form of CG,
// all of them in one persistent cooperative launch per residual-replacement cycle, FP64 reliable
// updates (residual replacement from the assembled FP64 CSR matrix) between the launches.
//
// Operator. The assembled matrix is the sum over the hexahedra c of kappa_c K_ref (the assembly keeps
// the element coefficients, in FP32, and K_ref). On an axis-aligned box the Q1 stiffness depends only
// on which coordinates of two corners differ: K_ref[i][j] = f[i ^ j] (corner bits x, y, z). So the
// coupling of vertex v to v + d (d in {-1, 0, 1}^3) is f[|dx| + 2 |dy| + 4 |dz|] times the sum of
// kappa over the cells that hold both vertices, and these sums come from the 2 x 2 coefficients of the
// cell layers below and above v: per layer two row sums in each direction and their total, and the
// four below + above pair sums. w_v = sum_t f[t] G_t, G_t the kappa-sum-weighted sum of z over the
// neighbours of type t: 35 FMAs and 14 adds per row, where the element form takes 72. The operator's
// input lives on a zero-padded vertex layout (one layer of zero vertices around the grid), the
// coefficients on a zero-padded cell layout, so no load is predicated. Dirichlet rows (unit rows,
// zero columns) are the rows of boundary vertices: the operator's input is zb = D_m r with D_m = 0
// there (their columns drop out) and the row itself is w_v = z_v = r_v.
//
// Iteration: p = z + beta p, s = w + beta s, x32 += alpha p, r -= alpha s, z = D r; w = A z;
// gamma = r.z, delta = z.w, rr = r.r -> beta, alpha. In the persistent kernel a thread owns a vertex
// column's chunk of z planes for the whole launch. It updates its rows (s, p and x32 in shared memory
// where they fit; r and w are its own, only zb is read by others), and after a grid barrier applies
// the operator to them with three planes of z and two layers of coefficients in registers; the
// exchange of the three sums is the second barrier, and every block adds the packets in block order
// (bit-identical scalars in every block). 128^3: 26.8 us per iteration with the update as a pass over
// padded arrays, two release barriers and a sum after the second, 20.5 like this. The kernel
// returns when a residual replacement is due (the iterated residual dropped 10x), the tolerance or
// max_iter is reached, or on breakdown; the host then runs the FP64 reliable update (x64 += x32,
// r = b - A x64 from the FP64 CSR matrix, stagnation guard) and launches it again, starting with the
// operator on the replaced residual. Every grid-barrier wait is bounded (GDT_ECUDA when one runs out).
#include <cmath>
#include <cstring>
#include <vector>

#include "exchange.cuh"

namespace gdt {
namespace {

constexpr int TH = 256;
// threads per block of the persistent kernel (one block per SM): 768 at 80 registers. 640 threads at 96
// registers measured slower (fewer columns in flight), as did 1024 threads at 64 registers with
// one-plane-ahead loads (28.6 against 27.8 us, in the first layout).
constexpr int MT = 768;
// residual replacement when the iterated residual's square dropped by this factor since the last one
// (10x in the residual norm; 100x saved 5 of 11 replacements at 128^3 but cost 10 % more iterations)
constexpr double kReplaceDrop2 = 1e-2;

struct MfState {
  double alpha, beta, gamma, gamma_prev, alpha_prev;
  double rr, rr0, rr_ref, tol2, drop;
  double aim;  // |r|^2 at which the iterated residual ends the solve
  int iter, max_iter, converged, flag, breakdown, updates, restarting, replaced_iter, misses, fresh;
};

__device__ __forceinline__ bool mf_stopped(const MfState* st) { return entry_flag(&st->converged) != 0; }

// After a replacement, rr the square of the true residual. Its difference to the iterated one is the rounding of
// x64, about the same after every replacement, so where that is not small beside the tolerance the
// iterated residual aims lower, by 1.5 of it and at most to half the tolerance. A true residual that
// misses the tolerance all the same restarts the direction once (the recurrence for alpha does not
// survive a replacement as large as the residual itself: at 128^3 and a tolerance 1.3 times the floor the
// iteration stagnated without) and aims for half of that. Otherwise a cycle that gained less than 2x on the
// true residual means that the FP32 operator is too far from the FP64 one for the sequence to continue;
// from then on each replacement restarts the direction and waits for a 1000x drop (restarted FP64
// refinement around FP32 CG).
__device__ __forceinline__ void mf3_replaced(MfState* st, double rr) {
  const double tol = st->tol2 * st->rr0;
  const bool missed = rr > tol && st->rr <= st->aim && !st->restarting && st->misses < 3;
  st->misses += missed ? 1 : 0;
  if (!missed && !st->restarting && rr > 0.25 * st->rr_ref) {
    st->restarting = 1;
    st->drop = 1e-6;
  }
  st->fresh = missed || st->restarting;
  const double cut = st->misses == 0 ? 1.0 : st->misses == 1 ? 0.25 : st->misses == 2 ? 0.0625 : 0.015625;
  st->aim = cut * fmax(0.25 * tol, tol - 1.5 * fmax(rr - st->rr, 0.0));
  st->rr_ref = rr;
  st->rr = rr;
  st->flag = 0;
  st->updates += 1;
  st->replaced_iter = st->iter;
  if (rr <= st->tol2 * st->rr0 || st->iter >= st->max_iter) st->converged = 1;
  if (!isfinite(rr)) {
    st->breakdown = 1;
    st->converged = 1;
  }
}

// Layouts. The operator's input zb: vertex (x, y, z), -1 <= x <= nx, at (x + 1) + PX (y + 1) + PXY (z + 1); the
// coefficients: cell (cx, cy, cz), -1 <= cx <= nx - 1, at (cx + 1) + CPX (cy + 1) + CPXY (cz + 1). Everything
// else (p, s, x32, r, w, D_m) is read and written only by the thread that owns the row, and stored by item
// (a vertex column's chunk of zlen planes): plane t of item i at t * items + i.
struct Mf3 {
  int nx, ny, nz;
  int PX;
  long long PXY;
  int CPX;
  long long CPXY;
  int ncol;      // nx * ny vertex columns
  int chunks;    // z chunks per column
  int zlen;      // planes per chunk
  int items;     // ncol * chunks
  float f[8];    // K_ref[i][j] = f[i ^ j]
  __device__ int vidx(int v) const {
    const int x = v % nx, y = (v / nx) % ny, z = v / ncol;
    return (x + 1) + PX * (y + 1) + int(PXY) * (z + 1);
  }
  __device__ int pidx(int v) const {
    const int c = v % ncol, z = v / ncol;
    return z % zlen * items + z / zlen * ncol + c;
  }
};

template <int V>
using Ph = std::integral_constant<int, V>;

// Weighted sums of one plane P of z (3 x 3 around the column) with one cell layer (2 x 2
// coefficients k, their row sums and total sm): u3 over the four diagonal neighbours, u1 over the x
// neighbours, u2 over the y neighbours, u0 the centre. A layer couples the plane below it and the
// plane above it; a row gets f3 u3 + f1 u1 + f2 u2 + f0 u0 ("same", the layer next to the row's own
// plane) and f7 u3 + f5 u1 + f6 u2 + f4 u0 ("cross", the layer between the row's plane and the
// neighbouring plane) from each (plane, layer) pair it touches.
struct U4 {
  float u3, u1, u2, u0;
};
__device__ __forceinline__ U4 plane_layer(const float (&P)[9], const float (&k)[4], const float (&sm)[5]) {
  U4 u;
  u.u3 = k[0] * P[0];
  u.u3 = fmaf(k[1], P[2], u.u3);
  u.u3 = fmaf(k[2], P[6], u.u3);
  u.u3 = fmaf(k[3], P[8], u.u3);
  u.u1 = fmaf(sm[1], P[5], sm[0] * P[3]);
  u.u2 = fmaf(sm[3], P[7], sm[2] * P[1]);
  u.u0 = sm[4] * P[4];
  return u;
}
__device__ __forceinline__ float same_of(const float (&f)[8], const U4& u) {
  return fmaf(f[0], u.u0, fmaf(f[2], u.u2, fmaf(f[1], u.u1, f[3] * u.u3)));
}
__device__ __forceinline__ float cross_of(const float (&f)[8], const U4& u) {
  return fmaf(f[4], u.u0, fmaf(f[6], u.u2, fmaf(f[5], u.u1, f[7] * u.u3)));
}

// w = A zb over rows z0 .. z1 - 1 of vertex column (x, y); accumulates r.z, z.w and r.r of those rows.
// Row z is the sum over the cell layers z - 1 and z of their pairs with the planes they touch: the
// layer z - 1 pairs (with planes z - 1 and z) are summed one step ahead into `carry`. The loads run two
// planes ahead: step z computes with plane z + 1 and layer z, loaded by step z - 1, while the loads of
// plane z + 2, layer z + 1 and r of row z + 1 are in flight, so a step does not wait a full L2 latency.
template <bool DIR>
// (w restrict: its stores do not alias the loads, so the next plane's loads may be issued before this
// plane's store; zb and r are read with plain coherent loads, never the read-only path: other blocks
// wrote them before the last grid barrier)
__device__ __forceinline__ void mf3_column(const Mf3& g, int x, int y, int z0, int z1, const float* __restrict__ kap,
                                           const float* zb, const float* r, float* __restrict__ w, int item,
                                           float& gam, float& del, float& rr) {
  const long long vb = (x + 1) + (long long)g.PX * (y + 1) + g.PXY;  // vertex (x, y, 0)
  const float* zc = zb + vb;
  // r and w of the item's rows, plane z at (z - z0) * items
  const float* rc = r + item;
  float* wc = w + item;
  const int items = g.items;
  const float* kc = kap + x + (long long)g.CPX * y + g.CPXY;  // cell (x - 1, y - 1, 0)
  const long long PX = g.PX, PXY = g.PXY, CPX = g.CPX, CPXY = g.CPXY;
  const bool colbnd = DIR && (x == 0 || y == 0 || x == g.nx - 1 || y == g.ny - 1);
  float f[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) f[t] = g.f[t];
  auto load_plane = [&](int z, float(&v)[9]) {
    const float* q = zc + z * PXY;
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = q[(k % 3 - 1) + (k / 3 - 1) * PX];
  };
  // the 2 x 2 coefficients of cell layer cz
  auto load_layer = [&](int cz, float(&k)[4]) {
    const float* q = kc + cz * CPXY;
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = __ldg(q + (j & 1) + (j >> 1) * CPX);
  };
  // their row sums over y (a = 0, 1), over x (b = 0, 1) and total
  auto layer_sums = [](const float(&k)[4], float(&sm)[5]) {
    sm[0] = k[0] + k[2];
    sm[1] = k[1] + k[3];
    sm[2] = k[0] + k[1];
    sm[3] = k[2] + k[3];
    sm[4] = sm[0] + sm[1];
  };
  float P[3][9], K[2][4];
  float carry, rnext;
  {
    float pm[9], km[4], sm[5];
    load_plane(z0 - 1, pm);
    load_plane(z0, P[0]);
    load_layer(z0 - 1, km);
    load_plane(z0 + 1, P[1]);  // z0 < z1 <= nz: at most the padding plane nz
    load_layer(z0, K[0]);
    rnext = rc[0];
    layer_sums(km, sm);
    carry = cross_of(f, plane_layer(pm, km, sm)) + same_of(f, plane_layer(P[0], km, sm));
  }
  auto step = [&](auto ph, int z) {
    constexpr int PH = decltype(ph)::value;
    const float(&pc)[9] = P[PH % 3];
    const float(&pn)[9] = P[(PH + 1) % 3];
    const float(&kl)[4] = K[PH % 2];
    const float rv = rnext;
    if (z + 1 < z1) {  // the next step's operands: plane z + 2 <= z1 <= nz, layer z + 1 <= nz - 1
      load_plane(z + 2, P[(PH + 2) % 3]);
      load_layer(z + 1, K[(PH + 1) % 2]);
      rnext = rc[(z + 1 - z0) * items];
    }
    float sl[5];
    layer_sums(kl, sl);
    const U4 uc = plane_layer(pc, kl, sl), un = plane_layer(pn, kl, sl);
    float wv = carry + (same_of(f, uc) + cross_of(f, un));
    carry = cross_of(f, uc) + same_of(f, un);
    float zv = pc[4];
    if (DIR && (colbnd || z == 0 || z == g.nz - 1)) {
      zv = rv;  // unit row: z = r (the diagonal is 1), w = z
      wv = rv;
    }
    wc[(z - z0) * items] = wv;
    gam = fmaf(rv, zv, gam);
    del = fmaf(zv, wv, del);
    rr = fmaf(rv, rv, rr);
  };
  int z = z0;
  for (; z + 6 <= z1; z += 6) {
    step(Ph<0>{}, z);
    step(Ph<1>{}, z + 1);
    step(Ph<2>{}, z + 2);
    step(Ph<3>{}, z + 3);
    step(Ph<4>{}, z + 4);
    step(Ph<5>{}, z + 5);
  }
  if (z < z1) step(Ph<0>{}, z++);
  if (z < z1) step(Ph<1>{}, z++);
  if (z < z1) step(Ph<2>{}, z++);
  if (z < z1) step(Ph<3>{}, z++);
  if (z < z1) step(Ph<4>{}, z++);
}

// the operator pass over the grid's (column, z chunk) items, grid-stride
template <bool DIR>
__device__ __forceinline__ void mf3_apply_items(const Mf3& g, const float* __restrict__ kap, const float* zb,
                                                const float* r, float* __restrict__ w, float& gam, float& del,
                                                float& rr) {
  const int stride = gridDim.x * blockDim.x;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < g.items; it += stride) {
    const int c = it % g.ncol, k = it / g.ncol;
    const int z0 = k * g.zlen, z1 = min(g.nz, z0 + g.zlen);
    mf3_column<DIR>(g, c % g.nx, c / g.nx, z0, z1, kap, zb, r, w, it, gam, del, rr);
  }
}

// ---------------------------------------------------------------------------- persistent kernel ---
enum { MF3_CONTINUE = 0, MF3_INIT = 1, MF3_REPLACE = 2 };

struct MfPArgs {
  Mf3 g;
  const float* kap;
  const float* dm;  // D_m: Jacobi inverse diagonal (or 1), 0 on Dirichlet rows
  float* p;
  float* s;
  float* x32;
  float* r;
  float* w;
  float* zb;
  MfState* st;
  ExchangeView ex;  // the whole grid
  int start;        // MF3_INIT / MF3_REPLACE: the first pass is the operator alone
};

// The solver scalars live in shared memory (thread 0 updates them after each reduction), so the
// registers go to the operator's planes.
struct MfScalars {
  double alpha, beta, gamma, gamma_prev, alpha_prev, rr;
  double inv_gamma, inv_alpha;  // of gamma_prev and alpha_prev of the next iteration
  double enough;                // |r|^2 at which the launch ends: replacement due, or the tolerance
  double total[3];
  float af, bf;  // alpha and beta as the update pass uses them (one conversion, by thread 0)
  int iter, max_iter, done, flag, brk;
};

// p = z + beta p, s = w + beta s, x32 += alpha p, r -= alpha s, zb = D_m r of the thread's rows (z = D r: D_m, or 1
// where D_m is 0 on a Dirichlet row). s, p and x32 of plane t at [t * step], from shared or global memory.
template <int SH>
__device__ __forceinline__ void mf3_update_items(const MfPArgs& a, float af, float bf, float* smem) {
  const int stride = gridDim.x * blockDim.x, items = a.g.items;
  int sbase = threadIdx.x;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < items; it += stride) {
    const int c = it % a.g.ncol, k = it / a.g.ncol;
    const int len = min(a.g.zlen, a.g.nz - k * a.g.zlen);
    const int per = a.g.zlen * MT * ((items + stride - 1) / stride);  // of one array in shared memory
    float* zc = a.zb + (c % a.g.nx + 1) + (long long)a.g.PX * (c / a.g.nx + 1) + a.g.PXY * (k * a.g.zlen + 1);
    auto at = [&](int var, float* g, int t) -> float& { return var < SH ? smem[var * per + sbase + t * MT] : g[t * items + it]; };
    constexpr int U = 4;
    auto rows = [&](int t0, auto n) {
      constexpr int N = decltype(n)::value;
      float r[N], w[N], d[N], s[N], p[N], x[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const int i = (t0 + u) * items + it;
        r[u] = a.r[i];
        w[u] = a.w[i];
        d[u] = __ldg(a.dm + i);
        s[u] = at(0, a.s, t0 + u);
        p[u] = at(1, a.p, t0 + u);
        x[u] = at(2, a.x32, t0 + u);
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float zt = d[u] != 0.f ? d[u] * r[u] : r[u];
        const float pn = fmaf(bf, p[u], zt), sn = fmaf(bf, s[u], w[u]);
        const float rn = fmaf(-af, sn, r[u]);
        at(0, a.s, t0 + u) = sn;
        at(1, a.p, t0 + u) = pn;
        at(2, a.x32, t0 + u) = fmaf(af, pn, x[u]);
        a.r[(t0 + u) * items + it] = rn;
        zc[(t0 + u) * a.g.PXY] = d[u] * rn;
      }
    };
    int t = 0;
    for (; t + U <= len; t += U) rows(t, Ph<U>{});
    for (; t < len; ++t) rows(t, Ph<1>{});
    sbase += a.g.zlen * MT;
  }
}

template <bool DIR, int SH>
__global__ void __launch_bounds__(MT, 1) k_mf3_persistent(const __grid_constant__ MfPArgs a) {
  __shared__ ExchangeShared<256> sh;
  __shared__ MfScalars sc;
  extern __shared__ __align__(16) float mf_smem[];
  MfState* st = a.st;
  if (mf_stopped(st)) return;
  if (threadIdx.x == 0) {
    sc.alpha = st->alpha;
    sc.beta = st->beta;
    sc.gamma = st->gamma;
    sc.gamma_prev = st->gamma_prev;
    sc.alpha_prev = st->alpha_prev;
    sc.rr = st->rr;
    sc.iter = st->iter;
    sc.max_iter = st->max_iter;
    // a replacement less than 4x above the tolerance would be followed by another one at it
    sc.enough = st->drop * st->rr_ref > 16.0 * st->aim ? st->drop * st->rr_ref : st->aim;
    sc.inv_gamma = a.start == MF3_REPLACE ? 1.0 / sc.gamma_prev : 0.0;
    sc.inv_alpha = a.start == MF3_REPLACE ? 1.0 / sc.alpha_prev : 0.0;
    sc.done = sc.flag = sc.brk = 0;
    sh.fault = 0;
  }
  // s, p and x32 of the thread's rows to shared memory
  const int stride = gridDim.x * blockDim.x, items = a.g.items;
  const int per = a.g.zlen * MT * ((items + stride - 1) / stride);
  auto exchange_rows = [&](bool in) {
    float* const g[3] = {a.s, a.p, a.x32};
    int sbase = threadIdx.x;
    for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < items; it += stride, sbase += a.g.zlen * MT) {
      const int len = min(a.g.zlen, a.g.nz - it / a.g.ncol * a.g.zlen);
#pragma unroll
      for (int v = 0; v < SH; ++v)
        for (int t = 0; t < len; ++t) {
          float& own = mf_smem[v * per + sbase + t * MT];
          if (in) own = g[v][t * items + it];
          else g[v][t * items + it] = own;
        }
    }
  };
  exchange_rows(true);
  __syncthreads();
  unsigned int epoch = 0;
  int pass = a.start;
  while (true) {
    if (pass == MF3_CONTINUE) {
      mf3_update_items<SH>(a, sc.af, sc.bf, mf_smem);
      // (zb is read by the neighbours; the reciprocals of the next scalars are formed while thread 0 waits)
      group_barrier(a.ex, epoch, sh, [&] {
        sc.inv_gamma = 1.0 / sc.gamma;
        sc.inv_alpha = 1.0 / sc.alpha;
      });
      if (sh.fault) break;
    }
    // w = A zb and the three dots
    float vf[3] = {0.f, 0.f, 0.f};
    mf3_apply_items<DIR>(a.g, a.kap, a.zb, a.r, a.w, vf[0], vf[1], vf[2]);
    const double t = group_exchange_f32<false>(a.ex, epoch, vf, sh);
    if (threadIdx.x < 96) {
      if ((threadIdx.x & 31) == 0) sc.total[threadIdx.x >> 5] = t;
      asm volatile("bar.sync 1, 96;" ::: "memory");
      if (threadIdx.x == 0) {
        const double gam = sc.total[0], del = sc.total[1], rrn = sc.total[2];
        if (pass == MF3_INIT) {
          sc.gamma_prev = gam;
          sc.beta = 0.0;
          sc.alpha = gam / del;
          sc.alpha_prev = sc.alpha;
        } else {
          if (pass == MF3_CONTINUE) {
            sc.gamma_prev = sc.gamma;
            sc.alpha_prev = sc.alpha;
          }
          sc.beta = (pass == MF3_REPLACE && st->fresh) ? 0.0 : gam * sc.inv_gamma;
          sc.alpha = gam / fma(-sc.beta * gam, sc.inv_alpha, del);
        }
        sc.gamma = gam;
        sc.af = float(sc.alpha);
        sc.bf = float(sc.beta);
        if (!(del > 0.0) || !isfinite(sc.alpha) || !isfinite(rrn)) {
          sc.brk = 1;
          sc.done = 1;
        } else if (pass == MF3_CONTINUE) {
          sc.iter += 1;
          sc.rr = rrn;
          if (rrn <= sc.enough || sc.iter >= sc.max_iter) {
            sc.flag = 1;
            sc.done = 1;
          }
        }
        if (sh.fault) sc.done = 1;
      }
    }
    __syncthreads();
    if (sc.done) break;
    pass = MF3_CONTINUE;
  }
  exchange_rows(false);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->alpha = sc.alpha;
    st->beta = sc.beta;
    st->gamma = sc.gamma;
    st->gamma_prev = sc.gamma_prev;
    st->alpha_prev = sc.alpha_prev;
    st->rr = sc.rr;
    st->iter = sc.iter;
    st->flag = sc.flag;
    if (sc.brk) {
      st->breakdown = 1;
      st->converged = 1;
    }
  }
}

// ------------------------------------------------------------------------------ setup kernels ---
// coefficients (lexicographic cells, FP32) into the padded cell layout
__global__ void k_mf3_cells(Mf3 g, const float* __restrict__ kin, float* __restrict__ kout) {
  const long long ncx = g.nx - 1, ncy = g.ny - 1, nc = ncx * ncy * (g.nz - 1);
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x) {
    const long long cx = c % ncx, cy = (c / ncx) % ncy, cz = c / (ncx * ncy);
    kout[(cx + 1) + g.CPX * (cy + 1) + g.CPXY * (cz + 1)] = kin[c];
  }
}

__device__ __forceinline__ bool on_boundary(const Mf3& g, int v) {
  const int x = v % g.nx, y = (v / g.nx) % g.ny, z = v / g.ncol;
  return x == 0 || y == 0 || z == 0 || x == g.nx - 1 || y == g.ny - 1 || z == g.nz - 1;
}

// D_m: 1 / diag (Jacobi) or 1, and 0 on the Dirichlet rows
__global__ void k_mf3_diag(int n, Mf3 g, const int* __restrict__ rp, const int* __restrict__ col,
                           const double* __restrict__ val, int jacobi, int dir, float* __restrict__ dm) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double d = 1.0;
    if (jacobi)
      for (int k = rp[i]; k < rp[i + 1]; ++k)
        if (col[k] == i) d = val[k];
    dm[g.pidx(i)] = (dir && on_boundary(g, i)) ? 0.f : float(1.0 / d);
  }
}

// probe of the operator against the assembled FP64 matrix: v(i) pseudo-random in [-1, 1]; r = v and
// zb = v with the Dirichlet rows' entries zeroed (the operator's input convention)
__device__ __forceinline__ double mf3_probe_value(long long i) {
  unsigned long long h = (unsigned long long)i * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 32;
  return double(h & 0xFFFFFF) / double(0x800000) - 1.0;
}

__global__ void k_mf3_probe(int n, Mf3 g, int dir, double* __restrict__ v64, float* __restrict__ r32,
                            float* __restrict__ zb) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = mf3_probe_value(i);
    v64[i] = v;
    r32[g.pidx(i)] = float(v);
    zb[g.vidx(i)] = (dir && on_boundary(g, i)) ? 0.f : float(v);
  }
}

template <bool DIR>
__global__ void __launch_bounds__(TH) k_mf3_apply(Mf3 g, const float* __restrict__ kap, const float* __restrict__ zb,
                                                 const float* __restrict__ r, float* __restrict__ w) {
  float a = 0.f, b = 0.f, c = 0.f;
  mf3_apply_items<DIR>(g, kap, zb, r, w, a, b, c);
}

// err[0] = max |A64 v - w|, err[1] = max |A64 v| (non-negative floats compare as their bit patterns)
template <int G, int PL>
__global__ void __launch_bounds__(TH) k_mf3_compare(int n, Mf3 g, const int* __restrict__ rp,
                                                   const int* __restrict__ col, const double* __restrict__ val,
                                                   const double* __restrict__ v64, const float* __restrict__ w,
                                                   unsigned int* err) {
  float md = 0.f, my = 0.f;
  for_rows_csr<G, PL, double>(n, rp, col, val, v64, [&](int row, bool leader, double y) {
    if (leader) {
      md = fmaxf(md, float(fabs(y - double(w[g.pidx(row)]))));
      my = fmaxf(my, float(fabs(y)));
    }
  });
  for (int o = 16; o > 0; o >>= 1) {
    md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, o));
    my = fmaxf(my, __shfl_xor_sync(0xffffffffu, my, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(err, __float_as_uint(md));
    atomicMax(err + 1, __float_as_uint(my));
  }
}

// the same check on the SELL-32 copy of the matrix
__global__ void __launch_bounds__(TH) k_mf3_compare_sell(SellView A, Mf3 g, const double* __restrict__ v64,
                                                        const float* __restrict__ w, unsigned int* err) {
  float md = 0.f, my = 0.f;
  for_slices(A, v64, [&](int row, bool active, double y, double) {
    if (active) {
      md = fmaxf(md, float(fabs(y - double(w[g.pidx(row)]))));
      my = fmaxf(my, float(fabs(y)));
    }
  });
  for (int o = 16; o > 0; o >>= 1) {
    md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, o));
    my = fmaxf(my, __shfl_xor_sync(0xffffffffu, my, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(err, __float_as_uint(md));
    atomicMax(err + 1, __float_as_uint(my));
  }
}

// start: r64 = b - A x (FP64), r32 = r64, zb = D_m r32; rr0
template <int G, int PL>
__global__ void __launch_bounds__(TH) k_mf3_init(int n, Mf3 g, const int* __restrict__ rp, const int* __restrict__ col,
                                                const double* __restrict__ val, const double* __restrict__ x,
                                                const double* __restrict__ b, float* __restrict__ r32,
                                                const float* __restrict__ dm, float* __restrict__ zb, MfState* st,
                                                double* partials, unsigned int* ticket) {
  double a1 = 0.0;
  for_rows_csr<G, PL, double>(n, rp, col, val, x, [&](int row, bool leader, double s) {
    if (leader) {
      const double ri = b[row] - s;
      const float rf = float(ri);
      const int ip = g.pidx(row);
      r32[ip] = rf;
      zb[g.vidx(row)] = dm[ip] * rf;
      a1 = fma(ri, ri, a1);
    }
  });
  double v[1] = {a1};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    st->rr = st->rr0 = st->rr_ref = v[0];
    st->drop = kReplaceDrop2;
    st->restarting = 0;
    st->aim = st->tol2 * v[0];
    st->misses = 0;
    st->fresh = 0;
    st->replaced_iter = -1;
    st->iter = 0;
    st->flag = 0;
    st->updates = 0;
    st->breakdown = 0;
    st->converged = (v[0] == 0.0) ? 1 : 0;
  }
}

// reliable update, part 1: x64 += x32, x32 = 0 (when a replacement is due, or always with `force`)
__global__ void __launch_bounds__(TH) k_mf3_accumulate(int n, Mf3 g, double* __restrict__ x, float* __restrict__ x32,
                                                      const MfState* st, int force) {
  if (!force && (mf_stopped(st) || !entry_flag(&st->flag))) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int ip = g.pidx(i);
    x[i] += double(x32[ip]);
    x32[ip] = 0.f;
  }
}

// reliable update, part 2: r64 = b - A64 x (FP64 CSR), r32 = r64, zb = D_m r32; convergence is decided
// on this true residual only
template <int G, int PL>
__global__ void __launch_bounds__(TH) k_mf3_true_residual(int n, Mf3 g, const int* __restrict__ rp,
                                                         const int* __restrict__ col, const double* __restrict__ val,
                                                         const double* __restrict__ x, const double* __restrict__ b,
                                                         float* __restrict__ r32, const float* __restrict__ dm,
                                                         float* __restrict__ zb, MfState* st, double* partials,
                                                         unsigned int* ticket) {
  if (mf_stopped(st) || !entry_flag(&st->flag)) return;
  double a1 = 0.0;
  for_rows_csr<G, PL, double>(n, rp, col, val, x, [&](int row, bool leader, double s) {
    if (leader) {
      const double ri = b[row] - s;
      const float rf = float(ri);
      const int ip = g.pidx(row);
      r32[ip] = rf;
      zb[g.vidx(row)] = dm[ip] * rf;
      a1 = fma(ri, ri, a1);
    }
  });
  double v[1] = {a1};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    mf3_replaced(st, v[0]);
  }
}

// the same two FP64 residual kernels on the SELL-32 copy of the matrix (where the SpMV schedule
// tuner picked it: one lane per row, coalesced entry loads)
__global__ void __launch_bounds__(TH) k_mf3_init_sell(SellView A, Mf3 g, const double* __restrict__ x,
                                                     const double* __restrict__ b, float* __restrict__ r32,
                                                     const float* __restrict__ dm, float* __restrict__ zb, MfState* st,
                                                     double* partials, unsigned int* ticket) {
  double a1 = 0.0;
  for_slices(A, x, [&](int row, bool active, double s, double) {
    if (active) {
      const double ri = b[row] - s;
      const float rf = float(ri);
      const int ip = g.pidx(row);
      r32[ip] = rf;
      zb[g.vidx(row)] = dm[ip] * rf;
      a1 = fma(ri, ri, a1);
    }
  });
  double v[1] = {a1};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    st->rr = st->rr0 = st->rr_ref = v[0];
    st->drop = kReplaceDrop2;
    st->restarting = 0;
    st->aim = st->tol2 * v[0];
    st->misses = 0;
    st->fresh = 0;
    st->replaced_iter = -1;
    st->iter = 0;
    st->flag = 0;
    st->updates = 0;
    st->breakdown = 0;
    st->converged = (v[0] == 0.0) ? 1 : 0;
  }
}

__global__ void __launch_bounds__(TH) k_mf3_true_residual_sell(SellView A, Mf3 g, const double* __restrict__ x,
                                                              const double* __restrict__ b, float* __restrict__ r32,
                                                              const float* __restrict__ dm, float* __restrict__ zb,
                                                              MfState* st, double* partials, unsigned int* ticket) {
  if (mf_stopped(st) || !entry_flag(&st->flag)) return;
  double a1 = 0.0;
  for_slices(A, x, [&](int row, bool active, double s, double) {
    if (active) {
      const double ri = b[row] - s;
      const float rf = float(ri);
      const int ip = g.pidx(row);
      r32[ip] = rf;
      zb[g.vidx(row)] = dm[ip] * rf;
      a1 = fma(ri, ri, a1);
    }
  });
  double v[1] = {a1};
  if (grid_reduce<1>(v, partials, ticket) && threadIdx.x == 0) {
    mf3_replaced(st, v[0]);
  }
}

// K_ref[i][j] = f[i ^ j] within FP32 rounding (axis-aligned boxes); false otherwise
bool xor_structure(const float* K, float* f) {
  float mx = 0.f;
  for (int k = 0; k < 64; ++k) mx = std::max(mx, std::fabs(K[k]));
  for (int t = 0; t < 8; ++t) f[t] = K[t];
  for (int i = 0; i < 8; ++i)
    for (int j = 0; j < 8; ++j)
      if (std::fabs(K[i * 8 + j] - f[i ^ j]) > 1e-6f * mx) return false;
  return mx > 0.f;
}

}  // namespace

bool mixed_mf_applies(gdt_matrix m) {
  const GridDesc& g = m->test.g;
  float f[8];
  return m->test.kind == GDT_SPACE_CG && m->test.order == 1 && g.dim == 3 && !g.simplex && m->mf_valid &&
         m->mf_kappa && m->rows == g.nvert && g.vn[0] >= 2 && g.vn[1] >= 2 && g.vn[2] >= 2 &&
         (g.vn[0] + 2) * (g.vn[1] + 2) * (g.vn[2] + 2) < (1LL << 31) && xor_structure(m->mf_K, f);
}

gdt_status solve_mixed_mf(gdt_context ctx, gdt_matrix m, const double* b, double* x, const gdt_solver_opts* o,
                          gdt_solve_info* info, cudaStream_t s) {
  const GridDesc& gd = m->test.g;
  const int n = int(m->rows);
  Mf3 g{};
  g.nx = int(gd.vn[0]);
  g.ny = int(gd.vn[1]);
  g.nz = int(gd.vn[2]);
  g.PX = g.nx + 2;
  g.PXY = (long long)g.PX * (g.ny + 2);
  g.CPX = g.nx + 1;
  g.CPXY = (long long)g.CPX * (g.ny + 1);
  g.ncol = g.nx * g.ny;
  if (!xor_structure(m->mf_K, g.f)) return GDT_EUNSUPPORTED;
  const long long ctot = g.CPXY * (g.nz + 1);
  const bool dir = m->mf_dirichlet != 0;
  const int vec_blocks = std::max(1, std::min(grid_blocks(n, TH), ctx->num_sms * 8));
  double* partials = ctx->scratch;
  unsigned int* ticket = ctx->counters;

  // persistent launch shape: one block of MT threads per SM (co-resident: cooperative launch)
  int coop = 0, per_sm = 0;
  GDT_TRY_CUDA(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
  if (!coop) return GDT_EUNSUPPORTED;
  int blocks = std::min(ctx->num_sms, 256);
  if (ctx->persistent_blocks > 0) blocks = std::min(blocks, ctx->persistent_blocks);
  // (column, z chunk) items: about one per thread
  const long long threads = (long long)blocks * MT;
  g.chunks = int(std::max(1LL, std::min<long long>(g.nz, threads / g.ncol)));
  g.zlen = (g.nz + g.chunks - 1) / g.chunks;
  g.chunks = (g.nz + g.zlen - 1) / g.zlen;
  if ((long long)g.ncol * g.chunks * g.zlen >= (1LL << 31)) return GDT_EUNSUPPORTED;
  g.items = g.ncol * g.chunks;
  // as many of s, p and x32 in shared memory as fit
  const long long per = 4LL * g.zlen * MT * ((g.items + threads - 1) / threads);
  const void* const fns[2][4] = {
      {reinterpret_cast<const void*>(&k_mf3_persistent<false, 0>), reinterpret_cast<const void*>(&k_mf3_persistent<false, 1>),
       reinterpret_cast<const void*>(&k_mf3_persistent<false, 2>), reinterpret_cast<const void*>(&k_mf3_persistent<false, 3>)},
      {reinterpret_cast<const void*>(&k_mf3_persistent<true, 0>), reinterpret_cast<const void*>(&k_mf3_persistent<true, 1>),
       reinterpret_cast<const void*>(&k_mf3_persistent<true, 2>), reinterpret_cast<const void*>(&k_mf3_persistent<true, 3>)}};
  long long room = 0;
  GDT_TRY_CUDA(ctx, allow_shared(ctx, fns[dir][3], &room));  // (all have the same static memory)
  const int shared = int(std::min(3LL, room / per));
  const void* fn = fns[dir][shared];
  const size_t dyn = size_t(shared * per);
  GDT_TRY_CUDA(ctx, allow_shared(ctx, fn, &room));
  GDT_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, MT, dyn));
  if (per_sm < 1) return GDT_EUNSUPPORTED;

  std::vector<void*> allocs;
  struct Freer {
    std::vector<void*>* a;
    cudaStream_t s;
    ~Freer() {
      for (void* p : *a) cudaFreeAsync(p, s);
    }
  } freer{&allocs, s};
  auto alloc = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (pool_malloc(ctx, &p, bytes + 256, s) != cudaSuccess) return nullptr;
    allocs.push_back(p);
    return reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
  };
  const size_t vb = sizeof(float) * size_t(g.items) * g.zlen, zbytes = sizeof(float) * size_t(g.PXY) * (g.nz + 2);
  float* p = (float*)alloc(vb);
  float* sv = (float*)alloc(vb);
  float* x32 = (float*)alloc(vb);
  float* r32 = (float*)alloc(vb);
  float* w = (float*)alloc(vb);
  float* zb = (float*)alloc(zbytes);
  float* dm = (float*)alloc(vb);
  float* kap = (float*)alloc(sizeof(float) * ctot);
  double* v64 = (double*)alloc(sizeof(double) * n);
  unsigned int* err = (unsigned int*)alloc(2 * sizeof(unsigned int));
  MfState* st = (MfState*)alloc(sizeof(MfState));
  if (!p || !sv || !x32 || !r32 || !w || !zb || !dm || !kap || !v64 || !err || !st)
    return fail(ctx, GDT_ENOMEM, "mixed solver vectors");
  for (float* v : {p, sv, x32}) GDT_TRY_CUDA(ctx, cudaMemsetAsync(v, 0, vb, s));
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(zb, 0, zbytes, s));
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(kap, 0, sizeof(float) * ctot, s));
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(err, 0, 2 * sizeof(unsigned int), s));
  MfState init{};
  init.tol2 = o->tol * o->tol;
  init.max_iter = o->max_iter;
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(st, &init, sizeof(MfState), cudaMemcpyHostToDevice, s));
  k_mf3_cells<<<vec_blocks, TH, 0, s>>>(g, m->mf_kappa, kap);
  k_mf3_diag<<<vec_blocks, TH, 0, s>>>(n, g, m->rp, m->col, m->val, o->precond == GDT_PREC_JACOBI, dir ? 1 : 0, dm);
  ctx->launches += 2;

  // the operator against the assembled FP64 matrix, one probe product (relative difference below 1e-4;
  // FP32 rounding is ~1e-6): values changed after assembly make the caller take the stencil path
  GDT_CHECK(ctx, tune_spmv(ctx, m));
  const LaunchShape sh = schedule_shape<double>(m->spmv_sched, n, ctx->num_sms);
  // the FP64 products (this check, the residuals) read the SELL-32 copy where the tuner chose it for
  // this matrix (the copy is refreshed here: the caller may have written the CSR values)
  const bool sell = m->use_sell && sell_prepare(ctx, m, s, true) == GDT_OK;
  const SellView SA = sell ? sell_view(m) : SellView{};
  {
    const int ablocks = int(std::min<long long>(((long long)g.ncol * g.chunks + TH - 1) / TH, 1LL << 30));
    k_mf3_probe<<<vec_blocks, TH, 0, s>>>(n, g, dir ? 1 : 0, v64, r32, zb);
    if (dir) k_mf3_apply<true><<<ablocks, TH, 0, s>>>(g, kap, zb, r32, w);
    else k_mf3_apply<false><<<ablocks, TH, 0, s>>>(g, kap, zb, r32, w);
#define GDT_MF3_COMPARE(GG, PP) \
  k_mf3_compare<GG, PP><<<sh.blocks, sh.threads, sh.smem, s>>>(n, g, m->rp, m->col, m->val, v64, w, err)
    if (sell)
      k_mf3_compare_sell<<<sell_blocks(SA.nslices, ctx->num_sms, reinterpret_cast<const void*>(&k_mf3_compare_sell)),
                           TH, 0, s>>>(SA, g, v64, w, err);
    else GDT_SCHEDULE_SWITCH(m->spmv_sched, GDT_MF3_COMPARE)
#undef GDT_MF3_COMPARE
    unsigned int herr[2] = {0u, 0u};
    GDT_TRY_CUDA(ctx, cudaMemcpyAsync(herr, err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    ctx->launches += 3;
    float ed, ey;
    std::memcpy(&ed, &herr[0], sizeof(float));
    std::memcpy(&ey, &herr[1], sizeof(float));
    if (!(ey > 0.f) || !std::isfinite(ed) || ed > 1e-4f * ey) return GDT_EUNSUPPORTED;
  }
  const int sblocks_init =
      sell ? sell_blocks(SA.nslices, ctx->num_sms, reinterpret_cast<const void*>(&k_mf3_init_sell)) : 0;
  const int sblocks =
      sell ? sell_blocks(SA.nslices, ctx->num_sms, reinterpret_cast<const void*>(&k_mf3_true_residual_sell)) : 0;
#define GDT_MF3_INIT(GG, PP)                                                                                     \
  k_mf3_init<GG, PP><<<sh.blocks, sh.threads, sh.smem, s>>>(n, g, m->rp, m->col, m->val, x, b, r32, dm, zb, st, \
                                                            partials, ticket)
  if (sell) k_mf3_init_sell<<<sblocks_init, TH, 0, s>>>(SA, g, x, b, r32, dm, zb, st, partials, ticket);
  else GDT_SCHEDULE_SWITCH(m->spmv_sched, GDT_MF3_INIT)
#undef GDT_MF3_INIT
  ctx->launches++;
  m->mx_operator = GDT_MIXED_OPERATOR_MATRIX_FREE;

  MfPArgs a{};
  a.g = g;
  a.kap = kap;
  a.dm = dm;
  a.p = p;
  a.s = sv;
  a.x32 = x32;
  a.r = r32;
  a.w = w;
  a.zb = zb;
  a.st = st;
  // fault flag and packets in the upper half of the scratch (kernels of the setup use its start)
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(ctx->scratch + kScratchDoubles / 2);
  const size_t packets = size_t(2 * kSlot) * blocks;
  static_assert(2 * kSlot * 256 + 16 <= kScratchDoubles / 2, "the packets fit the scratch");
  a.ex.fault = reinterpret_cast<unsigned int*>(words);
  a.ex.slots = words + 16;
  a.ex.first = 0;
  a.ex.count = blocks;
  a.ex.wait_ns = ctx->persistent_wait_ns > 0 ? (unsigned long long)ctx->persistent_wait_ns : kBarrierNs;
  MfState fin{};
  unsigned int fault = 0;
  int cycles = 0;
  // Cycles are enqueued four at a time and the host reads the state once per group: every kernel of a
  // cycle returns at entry once the solve has converged, so a group's surplus launches cost only their
  // launch, and the GPU does not idle for a host round trip after every replacement. The fault flag is
  // cleared once per solve: a barrier wait that runs out in any cycle stays visible, and the group's
  // remaining launches leave at their first barrier.
  constexpr int kCyclesPerCheck = 4;
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(a.ex.fault, 0, sizeof(unsigned int), s));
  while (cycles < 100000) {
    for (int k = 0; k < kCyclesPerCheck && cycles < 100000; ++k, ++cycles) {
      a.start = cycles == 0 ? MF3_INIT : MF3_REPLACE;
      GDT_TRY_CUDA(ctx, cudaMemsetAsync(a.ex.slots, 0, sizeof(unsigned long long) * packets, s));
      void* args[] = {&a};
      timing_begin(ctx, s, GDT_TIMING_MIXED_PERSISTENT);
      const cudaError_t le = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(MT), args, dyn, s);
      timing_end(ctx, s);
      GDT_TRY_CUDA(ctx, le);
      ctx->launches++;
      // the FP64 reliable update (both kernels return at once unless a replacement is due)
      timing_begin(ctx, s, GDT_TIMING_RELIABLE_UPDATE);
      k_mf3_accumulate<<<vec_blocks, TH, 0, s>>>(n, g, x, x32, st, 0);
#define GDT_MF3_TRUE_RESIDUAL(GG, PP)                                                                            \
  k_mf3_true_residual<GG, PP><<<sh.blocks, sh.threads, sh.smem, s>>>(n, g, m->rp, m->col, m->val, x, b, r32, dm, \
                                                                     zb, st, partials, ticket)
      if (sell) k_mf3_true_residual_sell<<<sblocks, TH, 0, s>>>(SA, g, x, b, r32, dm, zb, st, partials, ticket);
      else GDT_SCHEDULE_SWITCH(m->spmv_sched, GDT_MF3_TRUE_RESIDUAL)
#undef GDT_MF3_TRUE_RESIDUAL
      timing_end(ctx, s);
      ctx->launches += 2;
    }
    GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fin, st, sizeof(MfState), cudaMemcpyDeviceToHost, s));
    GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fault, a.ex.fault, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
    if (ctx->timing) timing_harvest(ctx);
    if (fault) return fail(ctx, GDT_ECUDA, "persistent mixed solver: a grid barrier wait ran out");
    if (fin.converged) break;
  }
  {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ctx, GDT_ECUDA, std::string("persistent mixed CG: ") + cudaGetErrorString(e));
  }
  gdt_solve_info res{};
  res.iterations = fin.iter;
  res.refinements = fin.updates;
  res.rel_residual = fin.rr0 > 0 ? std::sqrt(fin.rr / fin.rr0) : 0.0;
  res.converged = (!fin.breakdown && (fin.rr0 == 0 || fin.rr <= fin.tol2 * fin.rr0)) ? 1 : 0;
  if (info) *info = res;
  if (!res.converged) return fail(ctx, GDT_ENOCONV, "linear solver did not converge");
  return GDT_OK;
}

}  // namespace gdt
