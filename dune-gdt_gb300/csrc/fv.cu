// Finite volumes on structured cube grids (m = 1):
//   AdvectionFvOperator::apply (operators/advection-fv.hh:66-115) = LocalAdvectionFvCouplingOperator on
//   every inner/periodic intersection once (local/operators/advection-fv.hh:127-153), the boundary
//   treatments by extrapolation or by a boundary flux on the non-periodic sides (:187-457), with
//   NumericalLaxFriedrichsFlux (local/numerical-fluxes/lax-friedrichs.hh:61-87), NumericalUpwindFlux
//   (upwind.hh:61-73) or NumericalEngquistOsherFlux (engquist-osher.hh:72-103);
//   estimate_dt_for_hyperbolic_system (tools/hyperbolic.hh:38-86); explicit Euler
//   (test/instationary-eocstudies/base.hh:428-447) and ExplicitRungeKuttaTimeStepper with the SSP2
//   tableau (tools/timestepper/explicit-rungekutta.hh:82-97, 237-270), r = -1.
//
// GB300 design: an FP64 instruction holds a quarter of an SM for 64 cycles, also where it is predicated off, and that
// pipe, not HBM, bounds this update. So every face flux is computed exactly once per stage, with as few
// FP64 instructions as the flux allows (fv_face4: two for Burgers LF), and all selecting, comparing and
// sign handling runs on the integer pipe. The second SSP stage fuses u1 = u - dt k0, k1 = L(u1) and
// u_new = u + (k0 + k1)(-dt/2) into one pass: per step it reads u (twice) and k0 and writes k0 and
// u_new (40 bytes per cell). Boundary treatments are ghost states in the halo (extrapolation: the inside
// state, Dirichlet: the prescribed one), for which the face flux is the boundary flux, since
// g(u, v, n) = -g(v, u, -n) for all three fluxes; a prescribed flux, or none, is selected in place of the
// computed face. Kernels: 2D tiles (fv2d_tile), 3D tiles that march along z (fv3d_march) and 1D
// segments (fv1d_segment); grids with a single cell in some direction, and batches of many small 1D and 3D
// states (tiled_ok), take fv_apply_kernel.
// SSP-RK2 steps before (FP64 per face: three instructions; boundary fluxes and 1D / 3D in the generic
// form, each face twice) and now: 2048^2 Burgers LF 197 and 161 us, with inflow and outflow 359 and 161;
// 128 x 140 x 120 929 and 152; 100,000 cells 25 and 6.6; 120 x 97 with boundaries 28 and 7.1.
#include <cmath>
#include <limits>

#include <cub/device/device_reduce.cuh>

#include "internal.cuh"

namespace gdt {
namespace {

struct FvParams {
  int flux;       // GDT_FLUX_*
  int numflux;    // GDT_NUMFLUX_*
  double vel[3];
  double lf_inv_lambda;  // 0: local LF; else the reference's fixed lambda_ (coefficient 0.5 / lambda_)
  int bkind[6];          // per side (-x, +x, -y, +y, -z, +z): GDT_FV_BOUNDARY_*, or -1 for a periodic side
  double bval[6];
  // the tiled kernels' form of the flux, 4 g (see fv_face4)
  int form4;             // FORM4_*
  double lam2;           // Burgers LF: 2 lambda_ for a fixed lambda_, 0 for the local one
  double tu[3], tv[3];   // linear transport: 4 g = tu u + tv v (EO: each term only for a positive state)
  int bounded;           // some side has a boundary treatment
  double bflux4[6];      // 4 g in +e_k direction through a side with a prescribed flux (or none: 0)
};

enum { FORM4_BURGERS_LF, FORM4_BURGERS_LF_FIXED, FORM4_BURGERS_EO, FORM4_BURGERS_UPWIND, FORM4_TRANSPORT_LINEAR,
       FORM4_TRANSPORT_UPWIND, FORM4_TRANSPORT_EO };

__device__ __forceinline__ double f_of(const FvParams& p, double u, int d) {
  return p.flux == GDT_FLUX_BURGERS ? 0.5 * u * u : p.vel[d] * u;
}
__device__ __forceinline__ double df_of(const FvParams& p, double u, int d) {
  return p.flux == GDT_FLUX_BURGERS ? u : p.vel[d];
}

// numerical flux g(u, v, n) for the unit normal n = sgn e_k (sgn = +-1), u the state on the side n
// points away from
__device__ __forceinline__ double normal_flux(const FvParams& p, int dim, int k, double sgn, double u, double v) {
  if (p.numflux == GDT_NUMFLUX_LAX_FRIEDRICHS) {
    double lam;
    if (p.lf_inv_lambda != 0.0) {
      lam = 1.0 / p.lf_inv_lambda;  // coefficient (u - v) * 0.5 / lambda_
    } else if (p.flux == GDT_FLUX_BURGERS) {
      lam = fmax(fabs(u), fabs(v));
    } else {
      lam = 0.0;
      for (int d = 0; d < dim; ++d) lam = fmax(lam, fabs(p.vel[d]));
    }
    const double fsum = sgn * (f_of(p, u, k) + f_of(p, v, k));
    return 0.5 * fma(u - v, lam, fsum);
  }
  if (p.numflux == GDT_NUMFLUX_ENGQUIST_OSHER) {
    // f(0).n + int_0^u max(n.f'(s), 0) ds + int_0^v min(n.f'(s), 0) ds, each integral only for a
    // positive state (the reference integrates over [0, state] only then); in closed form for both
    // fluxes, f(0) = 0: Burgers n.f'(s) = sgn s, transport n.f'(s) = sgn v_k
    if (p.flux == GDT_FLUX_BURGERS) {
      if (sgn > 0.0) return u > 0.0 ? 0.5 * u * u : 0.0;
      return v > 0.0 ? -0.5 * v * v : 0.0;
    }
    const double a = sgn * p.vel[k];
    return (u > 0.0 ? u * fmax(a, 0.0) : 0.0) + (v > 0.0 ? v * fmin(a, 0.0) : 0.0);
  }
  const double w = (u + v) * 0.5;
  return sgn * df_of(p, w, k) > 0.0 ? sgn * f_of(p, u, k) : sgn * f_of(p, v, k);
}

// numerical flux across a face with unit normal +e_k, seen from the lower cell (value u) to the upper (v)
__device__ __forceinline__ double face_flux(const FvParams& p, int dim, int k, double u, double v) {
  return normal_flux(p, dim, k, 1.0, u, v);
}

// flux through the boundary face on `side` (2k: -e_k, 2k+1: +e_k) of a cell with value u, in the
// direction of the outer normal (what the boundary operator adds as g |I| / |E|)
__device__ __forceinline__ double boundary_flux(const FvParams& p, int dim, int side, double u) {
  const int kind = p.bkind[side];
  const int k = side >> 1;
  const double sgn = (side & 1) ? 1.0 : -1.0;
  if (kind == GDT_FV_BOUNDARY_EXTRAPOLATE) return normal_flux(p, dim, k, sgn, u, u);
  if (kind == GDT_FV_BOUNDARY_DIRICHLET) return normal_flux(p, dim, k, sgn, u, p.bval[side]);
  if (kind == GDT_FV_BOUNDARY_FLUX) return p.bval[side];
  return 0.0;  // GDT_FV_BOUNDARY_NONE on a non-periodic grid: no operator on this side
}

// flux in +e_k direction through the lower (upper = false) or upper boundary face of a cell
__device__ __forceinline__ double boundary_face_flux(const FvParams& p, int dim, int k, bool upper, double u) {
  const double g = boundary_flux(p, dim, 2 * k + (upper ? 1 : 0), u);
  return upper ? g : -g;
}

// The tiled kernels work with 4 g: the factors 1/2 of the flux formulas move into the 1/4 of the update
// coefficients (scaling by powers of two is exact) and the transport fluxes collapse to precomputed
// linear combinations.
// u > 0 on the bit pattern (false for NaN, as in the flux formulas)
__device__ __forceinline__ bool positive(double u) {
  return (unsigned long long)__double_as_longlong(u) - 1 < 0x7ffull << 52;
}
// 2 q for a square q >= 0 (or NaN) on its bit pattern: a normal number's exponent plus one, a subnormal's bits
// shifted, infinity where that overflows
__device__ __forceinline__ double twice(double q) {
  unsigned long long b = (unsigned long long)__double_as_longlong(q);
  constexpr unsigned long long one = 1ull << 52, inf = 0x7ffull << 52;
  if (b < one) b <<= 1;
  else if (b < inf - one) b += one;
  else if (b < inf) b = inf;
  return __longlong_as_double((long long)b);
}
// what a cell contributes to the faces besides its value: 2 u^2 (Burgers LF), u^2 (its fixed-lambda form) or 4 f(u)
// (Burgers upwind, EO)
__host__ __device__ constexpr bool uses_squares(int form) {
  return form == FORM4_BURGERS_LF || form == FORM4_BURGERS_LF_FIXED || form == FORM4_BURGERS_UPWIND ||
         form == FORM4_BURGERS_EO;
}
template <int FORM>
__device__ __forceinline__ double cell_square(double u) {
  return FORM == FORM4_BURGERS_LF_FIXED ? u * u : twice(u * u);
}

// m = the one of u, v of larger magnitude: sd = d or -d and sel = qu or qv by the table at fv_face4. In inline PTX:
// written in C++ the mask and comparison are recognised as fabs and a comparison of doubles and moved to the FP64
// pipe, two more instructions there per face (234 instead of 167 us a step on 2048^2).
__device__ __forceinline__ void burgers_lf_choose(double u, double v, double d, double qu, double qv, double& sd,
                                                  double& sel) {
  asm("{\n\t"
      ".reg .b64 a, b, m;\n\t"
      ".reg .pred first, negative, keep;\n\t"
      "and.b64 a, %2, 0x7fffffffffffffff;\n\t"
      "and.b64 b, %3, 0x7fffffffffffffff;\n\t"
      "setp.ge.s64 first, a, b;\n\t"
      "selp.b64 m, %2, %3, first;\n\t"
      "setp.lt.s64 negative, m, 0;\n\t"
      "xor.pred keep, first, negative;\n\t"
      "selp.b64 m, 0, 0x8000000000000000, keep;\n\t"
      "xor.b64 %0, %4, m;\n\t"
      "selp.b64 %1, %6, %5, negative;\n\t"
      "}"
      : "=l"(*reinterpret_cast<long long*>(&sd)), "=l"(*reinterpret_cast<long long*>(&sel))
      : "l"(__double_as_longlong(u)), "l"(__double_as_longlong(v)), "l"(__double_as_longlong(d)),
        "l"(__double_as_longlong(qu)), "l"(__double_as_longlong(qv)));
}

// 4 g(u, v, +e_k) with qu, qv = cell_square(u), (v).
// Burgers LF is u^2 + v^2 + 2 max(|u|, |v|) (u - v). With m the state of larger magnitude that is
//   2 u^2 + (u - v)^2 for m = u > 0,  2 v^2 - (u - v)^2 for m = u < 0,
//   2 u^2 - (u - v)^2 for m = v > 0,  2 v^2 + (u - v)^2 for m = v < 0:
// one subtraction and one FMA on the FP64 pipe, the choices on bit patterns (for non-negative doubles
// the integer order is the floating-point order).
template <int FORM>
__device__ __forceinline__ double fv_face4(const FvParams& p, int k, double u, double v, double qu, double qv) {
  if constexpr (FORM == FORM4_BURGERS_LF) {
    const double d = u - v;
    double sd, sel;
    burgers_lf_choose(u, v, d, qu, qv, sd, sel);
    return fma(sd, d, sel);
  } else if constexpr (FORM == FORM4_BURGERS_LF_FIXED) {
    return fma(p.lam2, u - v, qu + qv);
  } else if constexpr (FORM == FORM4_TRANSPORT_LINEAR) {
    return fma(p.tu[k], u, p.tv[k] * v);
  } else if constexpr (FORM == FORM4_TRANSPORT_UPWIND) {  // one of the states alone, whatever the other is
    return p.tu[k] != 0.0 ? p.tu[k] * u : p.tv[k] * v;
  } else if constexpr (FORM == FORM4_BURGERS_EO) {  // 4 * (u > 0 ? u^2 / 2 : 0)
    return positive(u) ? qu : 0.0;
  } else if constexpr (FORM == FORM4_TRANSPORT_EO) {
    return fma(p.tu[k], positive(u) ? u : 0.0, p.tv[k] * (positive(v) ? v : 0.0));
  } else {  // Burgers upwind: f'((u + v) / 2) > 0 ? 4 f(u) : 4 f(v)
    return positive(u + v) ? qu : qv;
  }
}

// ------------------------------------------------------------------------- generic (any dim) ---
// range[c] = sum over the 2d faces of c of +-flux * |I| / |E| (periodic neighbours, or the boundary
// treatment of the side)
__global__ void fv_apply_kernel(GridDesc g, FvParams p, long long nbatch, const double* __restrict__ u,
                                double* __restrict__ out, const double* __restrict__ ubase, double a_u1,
                                int mode, double* __restrict__ u_next, double dt_coef) {
  // mode 0: out = L(u); mode 1 (Euler): u_next = u - dt L(u); mode 2 (SSP stage 2, u1 = ubase + a_u1 * out):
  //   u_next = ubase + dt_coef * (k0 + L(u1)) with k0 = out
  const long long N = g.nelem;
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= N * nbatch) return;
  const long long b = idx / N, c = idx % N;
  const long long off = b * N;
  long long ci[3];
  cell_multi(g, c, ci);
  auto val = [&](long long cell) -> double {
    if (mode == 2) return fma(out[off + cell], a_u1, ubase[off + cell]);
    return u[off + cell];
  };
  const double uc = val(c);
  double acc = 0.0;
  for (int k = 0; k < g.dim; ++k) {
    double area = 1.0;
    for (int j = 0; j < g.dim; ++j)
      if (j != k) area *= g.h[j];
    double vol = 1.0;
    for (int j = 0; j < g.dim; ++j) vol *= g.h[j];
    const double coef = area / vol;
    if (p.bkind[2 * k] >= 0) {  // boundary treatments on both sides of direction k
      const double fl = ci[k] == 0 ? boundary_face_flux(p, g.dim, k, false, uc) : 0.0;
      const double fu = ci[k] == g.n[k] - 1 ? boundary_face_flux(p, g.dim, k, true, uc) : 0.0;
      long long cm[3] = {ci[0], ci[1], ci[2]}, cp[3] = {ci[0], ci[1], ci[2]};
      double lo = fl, hi = fu;
      if (ci[k] > 0) {
        cm[k] = ci[k] - 1;
        lo = face_flux(p, g.dim, k, val(cell_index(g, cm)), uc);
      }
      if (ci[k] < g.n[k] - 1) {
        cp[k] = ci[k] + 1;
        hi = face_flux(p, g.dim, k, uc, val(cell_index(g, cp)));
      }
      acc += coef * (hi - lo);
      continue;
    }
    long long cm[3] = {ci[0], ci[1], ci[2]}, cp[3] = {ci[0], ci[1], ci[2]};
    cm[k] = (ci[k] + g.n[k] - 1) % g.n[k];
    cp[k] = (ci[k] + 1) % g.n[k];
    const double um = val(cell_index(g, cm)), up = val(cell_index(g, cp));
    if (g.n[k] == 1) continue;  // a cell neighbouring itself has no flux
    acc += coef * (face_flux(p, g.dim, k, uc, up) - face_flux(p, g.dim, k, um, uc));
  }
  if (mode == 0) out[off + c] = acc;
  else if (mode == 1) u_next[off + c] = fma(-dt_coef, acc, u[off + c]);
  else u_next[off + c] = fma(dt_coef, out[off + c] + acc, ubase[off + c]);
}

// ------------------------------------------------------------------------------- tiled kernels ---
// One stage of a step. The fluxes are kept as 4 g, and the update as
// K = sum_k rho_k (g_k,upper - g_k,lower), rho_k = h_x / h_k, so that L(u) = K / (4 h_x):
//   STAGE 0: out = c_out K (fv_apply: c_out = 1 / (4 h_x), giving L(u)), or K itself for c_out = 1 (the first
//            SSP-RK2 stage: no multiply by one per cell)
//   STAGE 1 (Euler): out = u + c_out K, c_out = -dt / (4 h_x)
//   STAGE 2 (SSP-RK2): u1 = u + c1 k0 on the tile + halo (k0 = K(u), c1 = -dt / (4 h_x)),
//            out = u + c_out (k0 + K(u1)), c_out = -dt / (8 h_x)
// FORM: the numerical flux, compiled as straight-line code.
struct StageArgs {
  const double* u;
  const double* k0;
  double* out;
  double c1, c_out, rho[3];
};

// The stages of a step follow each other in the stream, each reading what the one before wrote. They are launched with
// programmatic serialisation: a stage's blocks may be placed while the last ones of the stage before still
// run, and wait here, before their first access to the state, until that stage is complete and visible.
__device__ __forceinline__ void fv_stage_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// lets the next stage's blocks be placed; near the end of a block, since blocks placed early crowd the SMs that are
// done first (60^3 cells: 42 us a step when called at the start, 25 here, 31 without)
__device__ __forceinline__ void fv_stage_ends() { asm volatile("griddepcontrol.launch_dependents;"); }

// cell c in -1 .. n (beyond a partial tile: further) of a direction -> the cell whose state it takes
__device__ __forceinline__ long long fv_cell(long long c, long long n, bool periodic) {
  if (c < 0) return periodic ? n - 1 : 0;
  if (c >= n) return periodic && c == n ? 0 : n - 1;
  return c;
}
template <int STAGE>
__device__ __forceinline__ double fv_load(const StageArgs& a, long long cell) {
  double v = a.u[cell];
  if (STAGE == 2) v = fma(a.k0[cell], a.c1, v);
  return v;
}
// the state beyond a side: prescribed, or what fv_cell chose
__device__ __forceinline__ double fv_ghost(const FvParams& p, int k, long long c, long long n, double v) {
  if (p.bounded && c < 0 && p.bkind[2 * k] == GDT_FV_BOUNDARY_DIRICHLET) return p.bval[2 * k];
  if (p.bounded && c >= n && p.bkind[2 * k + 1] == GDT_FV_BOUNDARY_DIRICHLET) return p.bval[2 * k + 1];
  return v;
}
// 4 g through the face below cell c of direction k, or the side's flux in its place
__device__ __forceinline__ bool fv_side_flux(int kind) {
  return kind == GDT_FV_BOUNDARY_FLUX || kind == GDT_FV_BOUNDARY_NONE;
}
__device__ __forceinline__ double fv_side(const FvParams& p, int k, long long c, long long n, double f) {
  if (p.bounded && c == 0 && fv_side_flux(p.bkind[2 * k])) return p.bflux4[2 * k];
  if (p.bounded && c == n && fv_side_flux(p.bkind[2 * k + 1])) return p.bflux4[2 * k + 1];
  return f;
}
template <int STAGE>
__device__ __forceinline__ void fv_store(const StageArgs& a, long long cell, double K) {
  if (STAGE == 0) {
    if (a.c_out == 1.0) a.out[cell] = K;  // (a branch: a selected product would still be computed)
    else a.out[cell] = a.c_out * K;
  } else if (STAGE == 1) a.out[cell] = fma(a.c_out, K, a.u[cell]);
  else a.out[cell] = fma(a.c_out, a.k0[cell] + K, a.u[cell]);
}

constexpr int TX = 32, BY = 8;  // tile TX x TY cells (TY: 32 or 8), block TX x BY threads

// 2D: a tile of TX x TY cells of state blockIdx.z. Every FP64 pass runs whole warps over 32 values: the tile
// interior column by column, the two halo columns and the 33rd x face of every row in passes of their
// own (a pass with one active lane costs the FP64 pipe as much as a full one).
template <int STAGE, int FORM, int TY>
__global__ void __launch_bounds__(TX* BY) fv2d_tile(const __grid_constant__ GridDesc g,
                                                    const __grid_constant__ FvParams p,
                                                    const __grid_constant__ StageArgs a) {
  constexpr bool SQ = uses_squares(FORM);
  __shared__ double s[TY + 2][TX + 2];             // staged state: s[j + 1][i + 1] = cell (x0 + i, y0 + j)
  __shared__ double q[SQ ? TY + 2 : 1][TX + 2];    // its cell_square
  __shared__ double gx[TY][TX + 1];                // gx[j][i]: x face between tile columns i - 1 and i
  __shared__ double gy[TY + 1][TX];                // gy[j][i]: y face between tile rows j - 1 and j
  const long long nx = g.n[0], ny = g.n[1];
  const long long off = (long long)blockIdx.z * nx * ny;
  const long long x0 = (long long)blockIdx.x * TX, y0 = (long long)blockIdx.y * TY;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const bool px = p.bkind[0] < 0, py = p.bkind[2] < 0;  // periodic directions
  const int rows = (int)min((long long)TY, ny - y0);
  fv_stage_begin();
  auto stage = [&](int j, int i) {
    const long long cx = x0 + i - 1, cy = y0 + j - 1;
    double v = fv_load<STAGE>(a, off + fv_cell(cy, ny, py) * nx + fv_cell(cx, nx, px));
    v = fv_ghost(p, 0, cx, nx, v);
    v = fv_ghost(p, 1, cy, ny, v);
    s[j][i] = v;
    if constexpr (SQ) q[j][i] = cell_square<FORM>(v);
  };
  for (int j = ty; j < rows + 2; j += BY) stage(j, tx + 1);  // interior columns
  {
    // the two halo columns, 2 (TY + 2) values, in the block's first warps
    const int e = ty * TX + tx;
    if (e < 2 * (TY + 2) && e % (TY + 2) < rows + 2) stage(e % (TY + 2), e < TY + 2 ? 0 : TX + 1);
  }
  __syncthreads();
  auto face = [&](int k, int j, int i, int jl, int il) {  // between staged cells (jl, il) and (j, i)
    double f;
    if constexpr (SQ) f = fv_face4<FORM>(p, k, s[jl][il], s[j][i], q[jl][il], q[j][i]);
    else f = fv_face4<FORM>(p, k, s[jl][il], s[j][i], 0.0, 0.0);
    return k == 0 ? fv_side(p, 0, x0 + i - 1, nx, f) : fv_side(p, 1, y0 + j - 1, ny, f);
  };
  for (int j = ty; j < rows; j += BY) gx[j][tx] = face(0, j + 1, tx + 1, j + 1, tx);
  if (ty == 0 && tx < rows) gx[tx][TX] = face(0, tx + 1, TX + 1, tx + 1, TX);  // the right face of every row
  for (int j = ty; j <= rows; j += BY) gy[j][tx] = face(1, j + 1, tx + 1, j, tx + 1);
  __syncthreads();
  fv_stage_ends();
  const long long gxi = x0 + tx;
  if (gxi >= nx) return;
  for (int j = ty; j < rows; j += BY) {
    const double K = fma(a.rho[1], gy[j + 1][tx] - gy[j][tx], gx[j][tx + 1] - gx[j][tx]);
    fv_store<STAGE>(a, off + (y0 + j) * nx + gxi, K);
  }
}

// 3D: a tile of MX x MY cells marches up a chunk of z planes. Each plane's state is staged with its halo, a thread
// holds the state of its own column at z and z + 1 and the flux through its lower z face; faces of the x
// and y directions are computed once and read by the neighbour through shared memory. The two barriers of
// a plane also separate its reads from the next plane's stores: the state is read before the second, the
// faces are written after the first.
constexpr int MX = 32, MY = 8;

template <int STAGE, int FORM>
__global__ void __launch_bounds__(MX* MY) fv3d_march(const __grid_constant__ GridDesc g,
                                                     const __grid_constant__ FvParams p,
                                                     const __grid_constant__ StageArgs a, int chunk, int chunks) {
  constexpr bool SQ = uses_squares(FORM);
  __shared__ double s[MY + 2][MX + 2];
  __shared__ double q[SQ ? MY + 2 : 1][MX + 2];
  __shared__ double gx[MY][MX + 1];
  __shared__ double gy[MY + 1][MX];
  const long long nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const long long off = (long long)(blockIdx.z / chunks) * nx * ny * nz;
  const long long x0 = (long long)blockIdx.x * MX, y0 = (long long)blockIdx.y * MY;
  const long long z0 = (long long)(blockIdx.z % chunks) * chunk, z1 = min(nz, z0 + chunk);
  const int tx = threadIdx.x, ty = threadIdx.y, e = ty * MX + tx;
  const bool px = p.bkind[0] < 0, py = p.bkind[2] < 0, pz = p.bkind[4] < 0;
  const int rows = (int)min((long long)MY, ny - y0);
  // the thread's own column and, in the first threads, one value of the halo ring (of MX or MY + 2 at each end)
  const long long own = fv_cell(y0 + ty, ny, py) * nx + fv_cell(x0 + tx, nx, px);
  int hj = -1, hi = 0;
  if (e < 2 * MX) {  // rows below and above
    hj = e < MX ? 0 : rows + 1;
    hi = tx + 1;
  } else if (e < 2 * MX + 2 * MY) {  // columns left and right
    const int h = e - 2 * MX;
    hj = h % MY + 1;
    hi = h < MY ? 0 : MX + 1;
    if (hj > rows) hj = -1;
  }
  const long long hx = x0 + hi - 1, hy = y0 + hj - 1;
  const long long halo = fv_cell(hy, ny, py) * nx + fv_cell(hx, nx, px);
  // the state of the thread's column in plane z (a column right of the grid, in a partial tile, holds the state
  // beyond the upper x side)
  auto column = [&](long long z) {
    double v = fv_load<STAGE>(a, off + fv_cell(z, nz, pz) * nx * ny + own);
    if (x0 + tx >= nx) v = fv_ghost(p, 0, x0 + tx, nx, v);
    return fv_ghost(p, 2, z, nz, v);
  };
  auto plane = [&](long long z) { return off + fv_cell(z, nz, pz) * nx * ny; };
  fv_stage_begin();
  const double lower = column(z0 - 1);
  double cur = column(z0);
  double ring = hj >= 0 ? fv_load<STAGE>(a, plane(z0) + halo) : 0.0;
  double qcur = SQ ? cell_square<FORM>(cur) : 0.0;
  double gz = fv_side(p, 2, z0, nz, fv_face4<FORM>(p, 2, lower, cur, SQ ? cell_square<FORM>(lower) : 0.0, qcur));
  for (long long z = z0; z < z1; ++z) {
    if (ty < rows) {  // (the row above a partial tile belongs to the ring)
      s[ty + 1][tx + 1] = cur;
      if constexpr (SQ) q[ty + 1][tx + 1] = qcur;
    }
    if (hj >= 0) {
      double v = fv_ghost(p, 0, hx, nx, ring);
      v = fv_ghost(p, 1, hy, ny, v);
      s[hj][hi] = v;
      if constexpr (SQ) q[hj][hi] = cell_square<FORM>(v);
    }
    // the next plane, in flight over the faces of this one
    const double next = column(z + 1);
    if (hj >= 0 && z + 1 < z1) ring = fv_load<STAGE>(a, plane(z + 1) + halo);
    __syncthreads();
    auto face = [&](int k, int j, int i, int jl, int il) {  // between staged cells (jl, il) and (j, i)
      double f;
      if constexpr (SQ) f = fv_face4<FORM>(p, k, s[jl][il], s[j][i], q[jl][il], q[j][i]);
      else f = fv_face4<FORM>(p, k, s[jl][il], s[j][i], 0.0, 0.0);
      return k == 0 ? fv_side(p, 0, x0 + i - 1, nx, f) : fv_side(p, 1, y0 + j - 1, ny, f);
    };
    if (ty < rows) {
      gx[ty][tx] = face(0, ty + 1, tx + 1, ty + 1, tx);
      gy[ty][tx] = face(1, ty + 1, tx + 1, ty, tx + 1);
    }
    if (ty == 0) {
      if (tx < rows) gx[tx][MX] = face(0, tx + 1, MX + 1, tx + 1, MX);
      gy[rows][tx] = face(1, rows + 1, tx + 1, rows, tx + 1);
    }
    const double qnext = SQ ? cell_square<FORM>(next) : 0.0;
    const double gup = fv_side(p, 2, z + 1, nz, fv_face4<FORM>(p, 2, cur, next, qcur, qnext));
    __syncthreads();
    if (z + 1 == z1) fv_stage_ends();
    if (x0 + tx < nx && ty < rows) {
      const double dxy = fma(a.rho[1], gy[ty + 1][tx] - gy[ty][tx], gx[ty][tx + 1] - gx[ty][tx]);
      fv_store<STAGE>(a, off + (z * ny + y0 + ty) * nx + x0 + tx, fma(a.rho[2], gup - gz, dxy));
    }
    gz = gup;
    cur = next;
    qcur = qnext;
  }
}

// 1D: a segment of SX cells, one per thread; a thread computes the face below its cell, the last one also the face
// above
constexpr int SX = 256;

template <int STAGE, int FORM>
__global__ void __launch_bounds__(SX) fv1d_segment(const __grid_constant__ GridDesc g,
                                                   const __grid_constant__ FvParams p,
                                                   const __grid_constant__ StageArgs a) {
  constexpr bool SQ = uses_squares(FORM);
  __shared__ double s[SX + 2], q[SQ ? SX + 2 : 1], gx[SX + 1];
  const unsigned int segments = (unsigned int)((g.n[0] + SX - 1) / SX);
  const long long nx = g.n[0], off = (long long)(blockIdx.x / segments) * nx;
  const long long x0 = (long long)(blockIdx.x % segments) * SX;
  const bool px = p.bkind[0] < 0;
  const int cells = (int)min((long long)SX, nx - x0);
  fv_stage_begin();
  for (int i = threadIdx.x; i < cells + 2; i += SX) {
    const long long c = x0 + i - 1;
    const double v = fv_ghost(p, 0, c, nx, fv_load<STAGE>(a, off + fv_cell(c, nx, px)));
    s[i] = v;
    if constexpr (SQ) q[i] = cell_square<FORM>(v);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= cells; i += SX) {
    double f;
    if constexpr (SQ) f = fv_face4<FORM>(p, 0, s[i], s[i + 1], q[i], q[i + 1]);
    else f = fv_face4<FORM>(p, 0, s[i], s[i + 1], 0.0, 0.0);
    gx[i] = fv_side(p, 0, x0 + i, nx, f);
  }
  __syncthreads();
  fv_stage_ends();
  if ((int)threadIdx.x < cells) fv_store<STAGE>(a, off + x0 + threadIdx.x, gx[threadIdx.x + 1] - gx[threadIdx.x]);
}

FvParams make_params(const GridDesc& g, const gdt_fv_desc* d) {
  FvParams p;
  p.flux = d->flux;
  p.numflux = d->numflux;
  for (int i = 0; i < 3; ++i) p.vel[i] = d->velocity[i];
  p.lf_inv_lambda = d->lf_lambda;
  p.lam2 = 0.0;
  p.bounded = 0;
  for (int k = 0; k < 3; ++k) p.tu[k] = p.tv[k] = 0.0;
  if (d->flux == GDT_FLUX_BURGERS) {
    if (d->numflux == GDT_NUMFLUX_LAX_FRIEDRICHS) {
      p.form4 = d->lf_lambda != 0.0 ? FORM4_BURGERS_LF_FIXED : FORM4_BURGERS_LF;
      p.lam2 = d->lf_lambda != 0.0 ? 2.0 / d->lf_lambda : 0.0;
    } else if (d->numflux == GDT_NUMFLUX_ENGQUIST_OSHER) {
      p.form4 = FORM4_BURGERS_EO;
    } else {
      p.form4 = FORM4_BURGERS_UPWIND;
    }
  } else {
    double lam = 0.0;
    for (int k = 0; k < g.dim; ++k) lam = std::max(lam, std::fabs(d->velocity[k]));
    if (d->lf_lambda != 0.0) lam = 1.0 / d->lf_lambda;
    p.form4 = d->numflux == GDT_NUMFLUX_ENGQUIST_OSHER ? FORM4_TRANSPORT_EO
              : d->numflux == GDT_NUMFLUX_UPWIND       ? FORM4_TRANSPORT_UPWIND
                                                       : FORM4_TRANSPORT_LINEAR;
    for (int k = 0; k < 3; ++k) {
      const double a = d->velocity[k];
      if (d->numflux == GDT_NUMFLUX_LAX_FRIEDRICHS) {  // 2 (a (u + v) + lambda (u - v))
        p.tu[k] = 2.0 * (a + lam);
        p.tv[k] = 2.0 * (a - lam);
      } else if (d->numflux == GDT_NUMFLUX_UPWIND) {  // 4 a u if a > 0 else 4 a v
        p.tu[k] = a > 0.0 ? 4.0 * a : 0.0;
        p.tv[k] = a > 0.0 ? 0.0 : 4.0 * a;
      } else {  // EO: 4 (u max(a, 0) + v min(a, 0)), each for a positive state
        p.tu[k] = 4.0 * std::max(a, 0.0);
        p.tv[k] = 4.0 * std::min(a, 0.0);
      }
    }
  }
  for (int side = 0; side < 6; ++side) {
    // a side is periodic when the grid is and no treatment is given; otherwise the treatment (or none)
    const bool periodic = g.periodic && d->boundary[side] == GDT_FV_BOUNDARY_NONE;
    p.bkind[side] = periodic ? -1 : d->boundary[side];
    p.bval[side] = d->boundary_value[side];
    if (side < 2 * g.dim && p.bkind[side] >= 0) p.bounded = 1;
    p.bflux4[side] = p.bkind[side] == GDT_FV_BOUNDARY_FLUX ? ((side & 1) ? 4.0 : -4.0) * p.bval[side] : 0.0;
  }
  return p;
}

// planes per block of fv3d_march: the chunk with the least work per SM, 13 FP64 instructions per cell of a plane, four
// for the face and the squares a chunk computes besides, its two plane loads before the first face counted
// as six more, and two chunks for what latency and the last wave leave idle (20 x 25 x 18 cells: 12.8 us a
// step with one plane, 29 with four; 60^3: 32 us with one or four, 25 with two; 128 x 140 x 120: 158 us
// with eight, 176 with fourteen)
int march_chunk(gdt_context ctx, const GridDesc& g, long long nbatch) {
  const double tiles = double((g.n[0] + MX - 1) / MX) * double((g.n[1] + MY - 1) / MY) * double(nbatch);
  double best = 0.0;
  int chosen = 1;
  for (int chunk = 1; chunk <= 16 && chunk <= g.n[2]; ++chunk) {
    const double blocks = tiles * double((g.n[2] + chunk - 1) / chunk);
    const double cost = (blocks / ctx->num_sms + 2.0) * (13 * chunk + 10);
    if (best == 0.0 || cost < best) best = cost, chosen = chunk;
  }
  return chosen;
}

// Whether the tiled kernels take the grid: at least two cells per direction (a cell that neighbours itself has no
// flux) and, in 1D and 3D, where the generic kernel takes any batch, as many blocks as a launch can have and less
// time. Many small states leave most of their tiles empty: a tile's warp computes 32 cells of a row whether
// they are there or not, the generic kernel each cell of the batch with every face twice. The estimates are of
// an SSP-RK2 step in us, from these (generic and tiled; 1D: 40,000 states, 3D: 8,000, then 1,000 states):
//   2 cells 25 and 89, 5 42 and 89, 10 72 and 88, 20 129 and 88, 64 387 and 99
//   2^3 41 and 173, 4^3 239 and 366, 5^3 436 and 498, 6^3 748 and 650; 2 x 64 x 2 123 and 288,
//   4 x 8 x 16 239 and 274, 8 x 8 x 2 74 and 42, 10^3 436 and 279, 32 x 4 x 4 240 and 58
// A few states take the tiles in any case (one of 4^3 19 and 6.5, 300 of them 25 and 19).
bool tiled_ok(gdt_context ctx, const GridDesc& g, long long nbatch) {
  for (int k = 0; k < g.dim; ++k)
    if (g.n[k] < 2) return false;
  const double cells = double(g.nelem) * double(nbatch);
  if (g.dim == 1) {
    const long long segments = (g.n[0] + SX - 1) / SX, last = g.n[0] - (segments - 1) * SX;
    const double warps = double(segments - 1) * (SX / 32) + double((last + 31) / 32);
    const double tiled = 4.6 + 1e-3 * double(nbatch) * (1.8 * double(segments) + 0.4 * warps);
    return segments * nbatch < (1LL << 31) && tiled <= std::max(14.5, 10.0 + 0.15e-3 * cells);
  }
  if (g.dim == 3) {
    const int chunk = march_chunk(ctx, g, nbatch);
    const long long tiles_x = (g.n[0] + MX - 1) / MX, tiles_y = (g.n[1] + MY - 1) / MY;
    const double plane = double(tiles_x) * (7.0 * double(tiles_y) + 1.4 * double(g.n[1]));
    const double tiled = 6.0 + 1e-3 * double(nbatch) * double(g.n[2]) * plane;
    return tiles_y <= 65535 && (g.n[2] + chunk - 1) / chunk * nbatch <= 65535 &&
           tiled <= std::max(24.7, 11.0 + 0.43e-3 * cells);
  }
  return true;
}

template <class... Args>
void launch_serial(cudaStream_t s, void (*kernel)(Args...), dim3 grid, dim3 block, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int STAGE, int FORM>
void launch_form(gdt_context ctx, const GridDesc& g, const FvParams& p, const StageArgs& a, long long nbatch) {
  cudaStream_t s = ctx->stream;
  if (g.dim == 2) {
    // Tiles of 32 rows compute 3 % of the faces twice, tiles of 8 rows 9 %, but a tile of 32 is 2 us of an SM's FP64
    // pipe: below two of them per SM the small ones share the work out better (SSP-RK2 steps, 32 and 8 rows:
    // 120 x 97 cells 17.0 and 12.8 us, 300 x 280 16.9 and 13.9, 512 x 500 21.1 and 21.0, 1000^2 47 and 50,
    // 2048^2 167 and 196)
    auto grid = [&](int rows) {
      return dim3((unsigned)((g.n[0] + TX - 1) / TX), (unsigned)((g.n[1] + rows - 1) / rows), (unsigned)nbatch);
    };
    const dim3 tall = grid(32), flat = grid(8);
    if ((long long)tall.x * tall.y * tall.z >= 2LL * ctx->num_sms || flat.y > 65535)
      launch_serial(s, &fv2d_tile<STAGE, FORM, 32>, tall, dim3(TX, BY), g, p, a);
    else launch_serial(s, &fv2d_tile<STAGE, FORM, 8>, flat, dim3(TX, BY), g, p, a);
  } else if (g.dim == 1) {
    launch_serial(s, &fv1d_segment<STAGE, FORM>, dim3((unsigned)((g.n[0] + SX - 1) / SX * nbatch)), dim3(SX), g, p, a);
  } else {
    const int chunk = march_chunk(ctx, g, nbatch);
    const int chunks = (int)((g.n[2] + chunk - 1) / chunk);
    const dim3 grid((unsigned)((g.n[0] + MX - 1) / MX), (unsigned)((g.n[1] + MY - 1) / MY), (unsigned)(nbatch * chunks));
    launch_serial(s, &fv3d_march<STAGE, FORM>, grid, dim3(MX, MY), g, p, a, chunk, chunks);
  }
}

// one stage of the tiled kernels, instantiated for the flux form
template <int STAGE>
void launch_stage(gdt_context ctx, const GridDesc& g, const FvParams& p, long long nbatch, const double* u,
                  const double* k0, double* out, double c1, double c_out) {
  StageArgs a;
  a.u = u;
  a.k0 = k0;
  a.out = out;
  a.c1 = c1;
  a.c_out = c_out;
  for (int k = 0; k < 3; ++k) a.rho[k] = k < g.dim ? g.h[0] / g.h[k] : 0.0;
  switch (p.form4) {
    case FORM4_BURGERS_LF: launch_form<STAGE, FORM4_BURGERS_LF>(ctx, g, p, a, nbatch); break;
    case FORM4_BURGERS_LF_FIXED: launch_form<STAGE, FORM4_BURGERS_LF_FIXED>(ctx, g, p, a, nbatch); break;
    case FORM4_BURGERS_EO: launch_form<STAGE, FORM4_BURGERS_EO>(ctx, g, p, a, nbatch); break;
    case FORM4_BURGERS_UPWIND: launch_form<STAGE, FORM4_BURGERS_UPWIND>(ctx, g, p, a, nbatch); break;
    case FORM4_TRANSPORT_LINEAR: launch_form<STAGE, FORM4_TRANSPORT_LINEAR>(ctx, g, p, a, nbatch); break;
    case FORM4_TRANSPORT_UPWIND: launch_form<STAGE, FORM4_TRANSPORT_UPWIND>(ctx, g, p, a, nbatch); break;
    default: launch_form<STAGE, FORM4_TRANSPORT_EO>(ctx, g, p, a, nbatch); break;
  }
}

}  // namespace

gdt_status fv_apply(gdt_context ctx, const gdt_space_s& sp, const gdt_fv_desc* d, const double* u, double* out) {
  const GridDesc& g = sp.g;
  FvParams p = make_params(g, d);
  if (tiled_ok(ctx, g, 1)) {
    launch_stage<0>(ctx, g, p, 1, u, nullptr, out, 0.0, 0.25 / g.h[0]);  // L(u) = K / (4 h_x)
  } else {
    fv_apply_kernel<<<grid_blocks(g.nelem, 256), 256, 0, ctx->stream>>>(g, p, 1, u, out, nullptr, 0.0, 0, nullptr,
                                                                        0.0);
  }
  return check_launch(ctx, "fv_apply");
}

gdt_status fv_estimate_dt(gdt_context ctx, const gdt_space_s& sp, const gdt_fv_desc* d, const double* u0,
                          double* dt) {
  // data range of the (elementwise constant) state, then the reference's formula on the host:
  // f' sampled at the Gauss points of order flux.order() on [min, max]; dt = 1 / (max |I|/|E| * max |f'|)
  const GridDesc& g = sp.g;
  cudaStream_t s = ctx->stream;
  double* dminmax = nullptr;
  GDT_TRY_CUDA(ctx, cudaMallocAsync(&dminmax, 2 * sizeof(double), s));
  size_t b1 = 0, b2 = 0;
  cub::DeviceReduce::Min(nullptr, b1, u0, dminmax, (int)g.nelem, s);
  cub::DeviceReduce::Max(nullptr, b2, u0, dminmax + 1, (int)g.nelem, s);
  void* tmp = nullptr;
  GDT_TRY_CUDA(ctx, cudaMallocAsync(&tmp, std::max(b1, b2), s));
  cub::DeviceReduce::Min(tmp, b1, u0, dminmax, (int)g.nelem, s);
  cub::DeviceReduce::Max(tmp, b2, u0, dminmax + 1, (int)g.nelem, s);
  double mm[2];
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(mm, dminmax, sizeof(mm), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaFreeAsync(tmp, s));
  GDT_TRY_CUDA(ctx, cudaFreeAsync(dminmax, s));
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  ctx->launches += 4;
  double data_minimum = std::min(std::numeric_limits<double>::max(), mm[0]);
  double data_maximum = std::max(std::numeric_limits<double>::min(), mm[1]);
  if (!(data_minimum < data_maximum)) data_maximum = data_minimum + 1e-6 * data_minimum;
  double max_df = std::numeric_limits<double>::min();
  // Gauss points on [0,1]: order 2 (Burgers) -> 2 points, order 1 (transport) -> 1 point
  const double g2 = 0.5 / std::sqrt(3.0);
  const double pts2[2] = {0.5 - g2, 0.5 + g2};
  const double pts1[1] = {0.5};
  const double* pts = d->flux == GDT_FLUX_BURGERS ? pts2 : pts1;
  const int npts = d->flux == GDT_FLUX_BURGERS ? 2 : 1;
  for (int q = 0; q < npts; ++q) {
    const double uq = data_minimum + (data_maximum - data_minimum) * pts[q];
    for (int ss = 0; ss < g.dim; ++ss) {
      const double df = d->flux == GDT_FLUX_BURGERS ? uq : d->velocity[ss];
      max_df = std::max(max_df, std::fabs(df));
    }
  }
  double vol = 1.0;
  for (int a = 0; a < g.dim; ++a) vol *= g.h[a];
  double perimeter = 0.0;
  for (int k = 0; k < g.dim; ++k) {
    double area = 1.0;
    for (int j = 0; j < g.dim; ++j)
      if (j != k) area *= g.h[j];
    perimeter += 2 * area;
  }
  const double pov = std::max(std::numeric_limits<double>::min(), perimeter / vol);
  *dt = 1.0 / (pov * max_df);
  return GDT_OK;
}

gdt_status fv_timestep(gdt_context ctx, const gdt_space_s& sp, const gdt_fv_desc* d, int stepper, double dt,
                       long long steps, long long nbatch, double* u, double* work) {
  // work holds 2 * nbatch * N doubles for SSP-RK2 (k0 and the next state), nbatch * N for Euler
  const GridDesc& g = sp.g;
  const FvParams p = make_params(g, d);
  cudaStream_t s = ctx->stream;
  const long long N = g.nelem * nbatch;
  double* cur = u;
  double* nxt = (stepper == GDT_TIMESTEPPER_SSPRK2) ? work + N : work;
  double* k0 = work;
  const bool tiled = tiled_ok(ctx, g, nbatch);
  // the tiled kernels' update K with L(u) = K / (4 h_x): the stepper keeps K0 = K(u) itself
  // (k0 = L(u) = K0 / (4 h_x)) and folds the factor into its coefficients
  const double ck = 0.25 / g.h[0];
  for (long long st = 0; st < steps; ++st) {
    if (stepper == GDT_TIMESTEPPER_EXPLICIT_EULER) {
      if (tiled)
        launch_stage<1>(ctx, g, p, nbatch, cur, nullptr, nxt, 0.0, -dt * ck);
      else
        fv_apply_kernel<<<grid_blocks(N, 256), 256, 0, s>>>(g, p, nbatch, cur, nullptr, nullptr, 0.0, 1, nxt, dt);
      ctx->launches++;
    } else {
      if (tiled) {
        launch_stage<0>(ctx, g, p, nbatch, cur, nullptr, k0, 0.0, 1.0);
        launch_stage<2>(ctx, g, p, nbatch, cur, k0, nxt, -dt * ck, -0.5 * dt * ck);
      } else {
        fv_apply_kernel<<<grid_blocks(N, 256), 256, 0, s>>>(g, p, nbatch, cur, k0, nullptr, 0.0, 0, nullptr, 0.0);
        fv_apply_kernel<<<grid_blocks(N, 256), 256, 0, s>>>(g, p, nbatch, nullptr, k0, cur, -dt, 2, nxt, -0.5 * dt);
      }
      ctx->launches += 2;
    }
    std::swap(cur, nxt);
  }
  {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ctx, GDT_ECUDA, std::string("fv_timestep: ") + cudaGetErrorString(e));
  }
  if (cur != u) GDT_TRY_CUDA(ctx, cudaMemcpyAsync(u, cur, sizeof(double) * N, cudaMemcpyDeviceToDevice, s));
  return GDT_OK;
}

}  // namespace gdt
