// Mixed-precision CG (FP32 CG with FP64 reliable updates, as mixed.cu) of structured vertex matrices as one
// cooperative launch: 1D, 2D and 3D P1/Q1 grids, mapped grids, matrices whose values changed after
// assembly. mixed.cu's graph form runs three kernels per iteration, each far below any limit of the
// chip at the sizes that fit here (303k rows of a mapped grid: 15.6 us of product, 34 us an iteration).
//
// A thread owns up to sixteen rows for the whole solve; x32, r, p, q and D^-1 of a row never leave its registers
// (p is also written for the neighbours). The FP32 matrix is stored by stencil slot (no column indices;
// 4 bytes an entry), a block keeps the slots of its slices that have a nonzero value in shared memory as
// far as it has room, and reads the rest from L2. Two exchanges (exchange.cuh) per iteration: beta comes
// from sums formed with q = A p (krylov.cu), so x, r and p are one pass. When a residual replacement is
// due, the same launch adds x32 to x, forms b - A x from the FP64 SELL copy and goes on with it; the
// decision is made beside the next product, which is then discarded (one product in forty).
#include <cmath>
#include <vector>

#include "exchange.cuh"
#include "structured.cuh"

namespace gdt {
namespace {

constexpr int MT = 512;      // threads per block (one block per SM)
constexpr int MW = MT / 32;  // warps
constexpr int MSLOTS = 27;

struct RState {
  double rr0, rr, tol2;
  int iter, max_iter, updates, converged, breakdown;
};

struct SlotOffsets {
  int count;
  int off[MSLOTS];  // distinct linear column offsets of a row, ascending
};

struct ResidentArgs {
  int n, nslices;
  SlotOffsets slots;
  const float* D;  // [slot][ld], row i of slot t at D[t * ld + i]
  long long ld;
  SellView A;      // the FP64 matrix
  const double* b;
  double* x;
  float* p;        // zeros below row 0 and above row n - 1
  int jacobi;
  RState* st;
  ExchangeView ex;
  int cap;         // FP32 entries a block may keep in shared memory
};

// row by slot from the CSR rows (both ascending)
__global__ void k_slot_matrix(int n, const int* __restrict__ rp, const int* __restrict__ col,
                              const double* __restrict__ val, SlotOffsets slots, float* __restrict__ D, long long ld,
                              int* __restrict__ bad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int t = 0;
    for (int k = rp[i]; k < rp[i + 1]; ++k) {
      const int o = col[k] - i;
      for (; t < slots.count && slots.off[t] < o; ++t) D[t * ld + i] = 0.f;
      if (t < slots.count && slots.off[t] == o) D[t++ * ld + i] = float(val[k]);
      else *bad = 1;
    }
    for (; t < slots.count; ++t) D[t * ld + i] = 0.f;
  }
}

struct ResidentShared {
  ExchangeShared<MT> ex;
  double total[3], last[2];
  double rho, rho_prev, stop, ref, drop, rr, rr0;
  float alpha, beta;
  int iter, updates, restarting, fresh, brk, conv;
  int go;  // 0: done, 1: next update, 2: replace the residual
};

// A row's product over the offsets listed for its slice, CH loads in flight (a whole 27-entry row where the registers
// allow it: with nine the rounds of one row waited for each other)
template <int CH, class LoadV>
__device__ __forceinline__ float slot_row(int w, const int* off, const float* p, LoadV v) {
  float s = 0.f;
#pragma unroll 1
  for (int t0 = 0; t0 < w; t0 += CH) {
    float vv[CH], pv[CH];
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      vv[j] = pv[j] = 0.f;
      if (t0 + j < w) {  // warp-uniform
        pv[j] = p[off[t0 + j]];
        vv[j] = v(t0 + j);
      }
    }
#pragma unroll
    for (int j = 0; j < CH; ++j) s = fmaf(vv[j], pv[j], s);
  }
  return s;
}

template <int R>
__global__ void __launch_bounds__(MT, 1) k_mixed_resident(const __grid_constant__ ResidentArgs a) {
  __shared__ ResidentShared sh;
  __shared__ int s_base[MW * R];                      // shared-memory offset of a slice's entries, -1: from D
  __shared__ unsigned char s_w[MW * R];               // nonzero slots of the slice
  __shared__ unsigned char s_slot[MW * R][MSLOTS + 1];  // which, and their column offsets
  __shared__ int s_off[MW * R][MSLOTS];
  constexpr int CH = R <= 4 ? MSLOTS : R <= 8 ? 14 : 9;
  extern __shared__ __align__(16) float mixed_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = int((long long)a.nslices * blockIdx.x / gridDim.x);
  const int ns = int((long long)a.nslices * (blockIdx.x + 1) / gridDim.x) - s0;
  if (threadIdx.x == 0) {
    sh.ex.fault = 0;
    sh.iter = sh.updates = sh.restarting = sh.brk = sh.conv = 0;
    sh.drop = 0.01;
  }
  auto local = [&](int k) { return warp + MW * k; };
  auto row_of = [&](int k) { return (s0 + local(k)) * 32 + lane; };
  // the nonzero slots of each slice
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int ls = local(k), row = row_of(k);
    int w = 0;
    if (ls < ns)
      for (int t = 0; t < a.slots.count; ++t) {
        const float v = row < a.n ? a.D[t * a.ld + row] : 0.f;
        if (__any_sync(0xffffffffu, v != 0.f)) {
          if (lane == 0) {
            s_slot[ls][w] = (unsigned char)t;
            s_off[ls][w] = a.slots.off[t];
          }
          ++w;
        }
      }
    if (lane == 0) s_w[ls] = (unsigned char)w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0;
    for (int ls = 0; ls < MW * R; ++ls) {
      const int need = 32 * s_w[ls];
      s_base[ls] = at + need <= a.cap ? at : -1;
      if (at + need <= a.cap) at += need;
    }
  }
  __syncthreads();
  float x[R], r[R], p[R], q[R], d[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int ls = local(k), row = row_of(k);
    x[k] = r[k] = p[k] = q[k] = d[k] = 0.f;
    if (ls < ns) {
      if (s_base[ls] >= 0)
        for (int t = 0; t < s_w[ls]; ++t)
          mixed_smem[s_base[ls] + 32 * t + lane] = row < a.n ? a.D[s_slot[ls][t] * a.ld + row] : 0.f;
    }
  }
  // b - A x of the thread's rows in FP64, with the sums over r32 D^-1 r32 and r^2
  auto true_residual = [&](float (&res)[R], double (&v)[2]) {
    v[0] = v[1] = 0.0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int ls = local(k), row = row_of(k);
      res[k] = 0.f;
      if (ls < ns) {
        const int2 md = __ldg(a.A.meta + s0 + ls);
        const double* gv = a.A.val + md.x + lane;
        const int* gc = a.A.col + md.x + lane;
        double s = 0.0;
#pragma unroll 1
        for (int t0 = 0; t0 < md.y; t0 += 9) {
          double vv[9], xv[9];
#pragma unroll
          for (int j = 0; j < 9; ++j) {
            vv[j] = xv[j] = 0.0;
            if (t0 + j < md.y) {
              vv[j] = __ldg(gv + 32 * (t0 + j));
              xv[j] = a.x[__ldg(gc + 32 * (t0 + j))];
            }
          }
#pragma unroll
          for (int j = 0; j < 9; ++j) s = fma(vv[j], xv[j], s);
        }
        if (row < a.n) {
          const double rd = a.b[row] - s;
          res[k] = float(rd);
          v[0] = fma(double(res[k]), double(d[k] * res[k]), v[0]);
          v[1] = fma(rd, rd, v[1]);
        }
      }
    }
  };
  unsigned int epoch = 0;
  // start: D^-1, r = b - A x, p = D^-1 r
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int ls = local(k), row = row_of(k);
    if (ls < ns && row < a.n) {
      double diag = 1.0;
      if (a.jacobi) {
        const int2 md = __ldg(a.A.meta + s0 + ls);
        for (int t = 0; t < md.y; ++t)
          if (__ldg(a.A.col + md.x + lane + 32 * t) == row) {  // (before the padding, which repeats the row's column)
            diag = __ldg(a.A.val + md.x + lane + 32 * t);
            break;
          }
      }
      d[k] = float(1.0 / diag);
    }
  }
  double v2[2];
  true_residual(r, v2);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    p[k] = d[k] * r[k];
    if (local(k) < ns && row_of(k) < a.n) a.p[row_of(k)] = p[k];
  }
  {
    const double t = group_exchange<true>(a.ex, epoch, v2, MW, sh.ex);
    if (threadIdx.x < 64 && lane == 0) sh.total[warp] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      sh.rho = sh.total[0];
      sh.rr = sh.rr0 = sh.ref = sh.total[1];
      sh.stop = a.st->tol2 * sh.rr0;
      sh.conv = sh.rr0 == 0.0;
      sh.go = !sh.conv && !sh.ex.fault;
    }
    __syncthreads();
  }
  bool pending = false;  // the sums of an update wait in sh.last
  while (sh.go) {
    float v3[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int ls = local(k);
      if (ls < ns) {  // warp-uniform
        const int row = row_of(k), base = s_base[ls], w = s_w[ls];
        const float* pr = a.p + row;
        if (base >= 0) {
          const float* sv = mixed_smem + base + lane;
          q[k] = slot_row<CH>(w, s_off[ls], pr, [&](int t) { return sv[32 * t]; });
        } else {
          const float* gv = a.D + row;
          const bool in = row < a.n;
          q[k] = slot_row<CH>(w, s_off[ls], pr, [&](int t) { return in ? __ldg(gv + s_slot[ls][t] * a.ld) : 0.f; });
        }
        const float dq = d[k] * q[k];
        v3[0] = fmaf(p[k], q[k], v3[0]);
        v3[1] = fmaf(r[k], dq, v3[1]);
        v3[2] = fmaf(q[k], dq, v3[2]);
      }
    }
    {
      const double t = group_exchange<false>(a.ex, epoch, v3, MW, sh.ex);
      if (threadIdx.x < 96) {
        const double inv = threadIdx.x == 0 ? 1.0 / t : 0.0;
        if (lane == 0) sh.total[warp] = t;
        asm volatile("bar.sync 1, 96;" ::: "memory");
        if (threadIdx.x == 0) {
          int go = 1;
          if (pending) {
            sh.rho_prev = sh.rho;
            sh.rho = sh.last[0];
            sh.rr = sh.last[1];
            sh.iter += 1;
            if (sh.rr <= sh.drop * sh.ref || sh.rr <= sh.stop || sh.iter >= a.st->max_iter) go = 2;
            if (!isfinite(sh.rr)) go = 0, sh.brk = 1;
          }
          if (go == 1) {
            if (!(t > 0.0) || !isfinite(t)) {
              go = 0;
              sh.brk = 1;
            } else {
              const double alpha = sh.rho * inv;
              sh.alpha = float(alpha);
              sh.beta = float(fma(alpha * inv, sh.total[2], fma(-2.0 * inv, sh.total[1], 1.0)));
            }
          }
          sh.go = sh.ex.fault ? 0 : go;
        }
      }
      __syncthreads();
    }
    if (!sh.go) break;
    if (sh.go == 2) {
      // replacement: x += x32, r = b - A x; p keeps its conjugate part (or restarts)
      pending = false;
#pragma unroll
      for (int k = 0; k < R; ++k)
        if (local(k) < ns && row_of(k) < a.n) a.x[row_of(k)] += double(x[k]);
      double none[1] = {0.0};
      group_exchange<true>(a.ex, epoch, none, 1, sh.ex);
      float res[R];
      true_residual(res, v2);
      const double t = group_exchange<false>(a.ex, epoch, v2, MW, sh.ex);
      if (threadIdx.x < 64 && lane == 0) sh.total[warp] = t;
      __syncthreads();
      if (threadIdx.x == 0) {
        // stagnation guard: a cycle that gained less than 2x on the true residual means the FP32 operator is
        // too far from the FP64 one for the sequence to continue; from then on each replacement restarts
        // the direction and waits for a 1000x drop (FP64 iterative refinement around FP32 CG)
        if (!sh.restarting && sh.total[1] > 0.25 * sh.ref) {
          sh.restarting = 1;
          sh.drop = 1e-6;
        }
        sh.ref = sh.rr = sh.total[1];
        sh.rho = sh.total[0];
        sh.updates += 1;
        // beta carries an absolute error of a few 1e-7 (its sums are of FP32 products): after a drop this steep in
        // one iteration that outweighs what it has to add, and the direction starts afresh
        sh.fresh = sh.restarting || sh.rho < 1e-5 * sh.rho_prev;
        if (sh.rr <= sh.stop || sh.iter >= a.st->max_iter) sh.conv = 1;
        if (!isfinite(sh.rr)) sh.brk = sh.conv = 1;
        sh.go = !sh.conv && !sh.ex.fault;
      }
      __syncthreads();
      if (!sh.go) break;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const float z = d[k] * res[k];
        p[k] = sh.fresh ? z : p[k] + (z - d[k] * r[k]);
        r[k] = res[k];
        x[k] = 0.f;
        if (local(k) < ns && row_of(k) < a.n) a.p[row_of(k)] = p[k];
      }
      group_exchange<true>(a.ex, epoch, none, 1, sh.ex);
      continue;
    }
    const float alpha = sh.alpha, beta = sh.beta;
    float v[2] = {0.f, 0.f};
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (local(k) < ns) {
        const int row = row_of(k);
        x[k] = fmaf(alpha, p[k], x[k]);
        r[k] = fmaf(-alpha, q[k], r[k]);
        const float z = d[k] * r[k];
        p[k] = fmaf(beta, p[k], z);
        if (row < a.n) a.p[row] = p[k];
        v[0] = fmaf(r[k], z, v[0]);
        v[1] = fmaf(r[k], r[k], v[1]);
      }
    const double t = group_exchange<true>(a.ex, epoch, v, MW, sh.ex);
    if (threadIdx.x < 64 && lane == 0) sh.last[warp] = t;
    pending = true;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.st->rr0 = sh.rr0;
    a.st->rr = sh.rr;
    a.st->iter = sh.iter;
    a.st->updates = sh.updates;
    a.st->converged = sh.conv;
    a.st->breakdown = sh.brk;
  }
}

}  // namespace

gdt_status solve_mixed_resident(gdt_context ctx, gdt_matrix m, const double* b, double* x, const gdt_solver_opts* o,
                                gdt_solve_info* info, cudaStream_t s) {
  const int n = int(m->rows);
  const GridDesc& g = m->test.g;
  int coop = 0;
  GDT_TRY_CUDA(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device));
  if (!coop) return GDT_EUNSUPPORTED;
  int blocks = std::min(ctx->num_sms, MT);
  if (ctx->persistent_blocks > 0) blocks = std::min(blocks, ctx->persistent_blocks);
  const int nslices = (n + 31) / 32;
  blocks = std::max(1, std::min(blocks, (nslices + 3) / 4));
  const int per_warp = ((nslices + blocks - 1) / blocks + MW - 1) / MW;
  // the distinct column offsets of the vertex stencil, ascending
  ResidentArgs a;
  std::vector<long long> offs;
  for (int k = 0; k < pow3(g.dim); ++k) {
    if (!slot_in_stencil(g.dim, g.simplex != 0, k)) continue;
    long long off = 0, stride = 1;
    for (int d = 0; d < g.dim; ++d) {
      off += slot_offset(k, d) * stride;
      stride *= g.vn[d];
    }
    offs.push_back(off);
  }
  std::sort(offs.begin(), offs.end());
  offs.erase(std::unique(offs.begin(), offs.end()), offs.end());
  a.slots.count = int(offs.size());
  for (size_t k = 0; k < offs.size(); ++k) a.slots.off[k] = int(offs[k]);
  const long long pad = (offs.back() + 63) / 64 * 64 + 32;  // and the unused lanes of the last slice
  // Sixteen rows per thread only for the short stencils: 1.2 M rows of P1 tetrahedra (seven nonzero slots) 31.2 ms in
  // mixed.cu's graph form and 20.2 here, but 1.05 M of mapped Q1 (27 slots, 113 MB streamed per product) 36.2
  // and 38.3. Up to eight rows the 27-slot stencils gain too: 303k rows 16.7 and 6.5 ms, 505k 21.8 and 12.1.
  const bool sixteen = a.slots.count <= 15;
  const void* fn = per_warp <= 1   ? reinterpret_cast<const void*>(&k_mixed_resident<1>)
                   : per_warp <= 2 ? reinterpret_cast<const void*>(&k_mixed_resident<2>)
                   : per_warp <= 4 ? reinterpret_cast<const void*>(&k_mixed_resident<4>)
                   : per_warp <= 8 ? reinterpret_cast<const void*>(&k_mixed_resident<8>)
                   : per_warp <= 16 && sixteen ? reinterpret_cast<const void*>(&k_mixed_resident<16>)
                                    : nullptr;
  if (!fn) return GDT_EUNSUPPORTED;  // more rows than the registers of the grid hold
  {
    // the values are copied at every solve: the caller may have written them through the CSR pointer
    const gdt_status ss = sell_prepare(ctx, m, s, true);
    if (ss != GDT_OK) return ss;
  }
  long long room = 0;
  GDT_TRY_CUDA(ctx, allow_shared(ctx, fn, &room));
  const long long want = 32LL * a.slots.count * ((nslices + blocks - 1) / blocks);
  a.cap = int(std::max(0LL, std::min(want, room / 4 / 32 * 32)));
  const size_t dyn = size_t(a.cap) * 4;
  int per_sm = 0;
  GDT_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, MT, dyn));
  if (per_sm < 1) return GDT_EUNSUPPORTED;
  a.n = n;
  a.nslices = nslices;
  a.ld = (n + 31) / 32 * 32;
  a.A = sell_view(m);
  a.b = b;
  a.x = x;
  a.jacobi = o->precond == GDT_PREC_JACOBI;
  const size_t plen = size_t(2 * pad + a.ld);
  struct Buffers {
    void* p[4] = {};
    cudaStream_t s;
    ~Buffers() {
      for (void* q : p)
        if (q) cudaFreeAsync(q, s);
    }
  } buf;
  buf.s = s;
  if (pool_malloc(ctx, &buf.p[0], sizeof(float) * a.ld * a.slots.count, s) != cudaSuccess ||
      pool_malloc(ctx, &buf.p[1], sizeof(float) * plen, s) != cudaSuccess ||
      pool_malloc(ctx, &buf.p[2], sizeof(RState), s) != cudaSuccess ||
      pool_malloc(ctx, &buf.p[3], sizeof(int), s) != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, GDT_ENOMEM, "mixed solver vectors");
  }
  a.D = static_cast<float*>(buf.p[0]);
  a.p = static_cast<float*>(buf.p[1]) + pad;
  a.st = static_cast<RState*>(buf.p[2]);
  int* const bad = static_cast<int*>(buf.p[3]);
  RState init{};
  init.tol2 = o->tol * o->tol;
  init.max_iter = o->max_iter;
  unsigned long long* const words = reinterpret_cast<unsigned long long*>(ctx->scratch + kScratchDoubles / 2);
  const size_t packets = size_t(2 * kSlot) * blocks;
  if (packets + 16 > kScratchDoubles / 2) return GDT_EUNSUPPORTED;
  a.ex.slots = words + 16;
  a.ex.fault = reinterpret_cast<unsigned int*>(words);
  a.ex.first = 0;
  a.ex.count = blocks;
  a.ex.wait_ns = ctx->persistent_wait_ns > 0 ? (unsigned long long)ctx->persistent_wait_ns : kBarrierNs;
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(words, 0, sizeof(unsigned long long) * (packets + 16), s));
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(buf.p[1], 0, sizeof(float) * plen, s));
  GDT_TRY_CUDA(ctx, cudaMemsetAsync(bad, 0, sizeof(int), s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(a.st, &init, sizeof(RState), cudaMemcpyHostToDevice, s));
  k_slot_matrix<<<std::max(1, std::min(grid_blocks(n, 256), ctx->num_sms * 8)), 256, 0, s>>>(
      n, m->rp, m->col, m->val, a.slots, static_cast<float*>(buf.p[0]), a.ld, bad);
  ctx->launches++;
  void* args[] = {&a};
  const cudaError_t le = cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(MT), args, dyn, s);
  if (le == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs available than the device has
    cudaGetLastError();
    return GDT_EUNSUPPORTED;
  }
  GDT_TRY_CUDA(ctx, le);
  ctx->launches++;
  RState fin;
  int hbad = 0;
  unsigned int fault = 0;
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fin, a.st, sizeof(RState), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaMemcpyAsync(&fault, a.ex.fault, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
  GDT_TRY_CUDA(ctx, cudaStreamSynchronize(s));
  if (fault) return fail(ctx, GDT_ECUDA, "persistent solver: a grid barrier wait ran out");
  if (hbad) return fail(ctx, GDT_EUNSUPPORTED, "matrix entry outside the vertex stencil");
  m->mx_operator = GDT_MIXED_OPERATOR_STENCIL;
  gdt_solve_info res{};
  res.iterations = fin.iter;
  res.refinements = fin.updates;
  res.rel_residual = fin.rr0 > 0 ? std::sqrt(fin.rr / fin.rr0) : 0.0;
  res.converged = (!fin.breakdown && (fin.rr0 == 0 || fin.rr <= o->tol * o->tol * fin.rr0)) ? 1 : 0;
  if (info) *info = res;
  if (!res.converged) return fail(ctx, GDT_ENOCONV, "linear solver did not converge");
  return GDT_OK;
}

}  // namespace gdt
