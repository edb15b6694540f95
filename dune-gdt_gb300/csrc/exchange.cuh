// Sums over a group of co-resident blocks that are also the group's barrier, for persistent kernels.
#pragma once
#include "linalg.cuh"

namespace gdt {

// One exchange is a sum of up to three values per thread and the barrier of the group in one: the block sums go
// out as one 32-byte packet, four words of 48 payload bits each beside 16 bits of the number of the
// sum, and every block polls the packets of its group until their words carry that number. All blocks
// add the packets in the same order, so all hold the same bits and none has to broadcast a decision. Two
// packet buffers alternate: a block can only write sum k + 2 after all have written k + 1, that is after
// all have read k.
// Polls delay the stores to the line they read, so a block's packet has 256 bytes of its own (152 blocks
// exchange in 0.98 us like that, in 2.4 us with packets of 16 bytes side by side) and is read once, not
// once per value (three values: 3.3 us with a packet and a polling warp each).
// An FP64 instruction occupies a quarter of the SM for 64 cycles, whichever warp issues it. So the block sums
// are formed by one warp per value from the threads' values in shared memory (a shuffle tree in every
// warp would issue five instructions for each one of these).
// Every wait is bounded (time and count); a wait that runs out sets the fault flag, which the callers
// check after every exchange.
constexpr int kSlot = 32;  // 64-bit words per block and buffer

struct ExchangeView {
  unsigned long long* slots;   // kSlot words per block of the grid, twice (zero before the launch)
  unsigned int* fault;         // set when a wait ran out (zero before the launch)
  unsigned long long wait_ns;  // longest wait
  int first, count;            // the blocks of the group: first .. first + count - 1
};

template <int T>
struct ExchangeShared {
  double part[3][T];
  double packet[3][T];  // of block first + b at [..][b]; cluster_exchange: [epoch & 1][3][16], written by the blocks
  double own[3];
  int fault;  // set by the caller to 0 before the first exchange
};

// lane l of a warp: v[l] + v[32 + l] + ..., then over the lanes, in a fixed order
__device__ __forceinline__ double sum_strided(const double* v, int groups) {
  double s[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = j < groups ? v[32 * j] : 0.0;
#pragma unroll 1
  for (int j0 = 4; j0 < groups; j0 += 4)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j0 + j < groups) s[j] += v[32 * (j0 + j)];
  double b = s[0];
  if (groups > 2) b = (s[0] + s[1]) + (s[2] + s[3]);
  else if (groups > 1) b = s[0] + s[1];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  return b;
}

// The same for FP32 values of the threads. A lane's are added with Knuth's two-sum, which gives the rounding error of
// every addition, so its sum is held in two words (16 random values: off by 2^-45 of their magnitudes at most, 2^-51
// on average) and the rest is FP64. Converted and added in FP64 from the first value on they cost 0.7 us in
// each of the two sums of an iteration (mapped Q1 of 67 x 60 x 72: 6.85 ms, 6.16 like this and with FP32 sums
// over a warp).
__device__ __forceinline__ double sum_strided(const float* v, int groups) {
  float s = groups > 0 ? v[0] : 0.f, e = 0.f;
#pragma unroll 4
  for (int j = 1; j < groups; ++j) {
    const float x = v[32 * j], t = s + x, y = t - s;
    e += (s - (t - y)) + (x - y);
    s = t;
  }
  double b = double(s) + double(e);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
  return b;
}

// The group's sums of what the block's threads have stored in sh.part[k][32 g + lane] (k < NV, g < groups), returned in
// all lanes of warp k for value k. RELEASE: the block's writes before the call are visible to the group's
// blocks after their next block barrier; without it only the order of their reads before the call and
// this block's writes after it is kept. At most T blocks; the epoch counts the group's exchanges.
// V: the type of the values stored in sh.part's memory.
template <bool RELEASE, int NV, class V, int T>
__device__ __forceinline__ double exchange_stored(const ExchangeView& ex, unsigned int& epoch, int groups,
                                                  ExchangeShared<T>& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ++epoch;
  __syncthreads();
  if (ex.count == 1) {
    const double b = warp < NV ? sum_strided(reinterpret_cast<const V*>(sh.part[warp]) + lane, groups) : 0.0;
    __syncthreads();  // part is free for the next exchange
    return b;
  }
  unsigned long long* const base = ex.slots + (size_t)kSlot * (gridDim.x * (epoch & 1u) + ex.first);
  const unsigned long long tag = (unsigned long long)epoch << 48;
  if (warp < NV) {
    const double b = sum_strided(reinterpret_cast<const V*>(sh.part[warp]) + lane, groups);
    if (lane == 0) sh.own[warp] = b;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * NV) : "memory");
    if (threadIdx.x == 0) {
      unsigned long long w[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) w[k] = k < NV ? __double_as_longlong(sh.own[k]) : 0ull;
      if (RELEASE) fence_acq_rel_gpu();
      asm volatile("st.relaxed.gpu.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(base + kSlot * (blockIdx.x - ex.first)),
                   "l"((w[0] & 0xffffffffffffull) | tag), "l"((w[0] >> 48) | ((w[1] & 0xffffffffull) << 16) | tag),
                   "l"((w[1] >> 32) | ((w[2] & 0xffffull) << 32) | tag), "l"((w[2] >> 16) | tag)
                   : "memory");
    }
  }
  if (warp * 32 < ex.count) {
    unsigned long long w[4] = {0, 0, 0, 0}, t0 = 0;
    bool wait = (int)threadIdx.x < ex.count;
    for (unsigned int spins = 1;; ++spins) {
      if (wait) {
        if (RELEASE)
          asm volatile("ld.acquire.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                       : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                       : "l"(base + kSlot * threadIdx.x)
                       : "memory");
        else
          asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                       : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                       : "l"(base + kSlot * threadIdx.x)
                       : "memory");
        wait = (((w[0] ^ tag) | (w[1] ^ tag) | (w[2] ^ tag) | (w[3] ^ tag)) >> 48) != 0;
      }
      if (!__any_sync(0xffffffffu, wait)) break;
      if (spins == 1u) t0 = global_ns();
      else if (spins == 2u || (spins & 255u) == 0u) {
        const bool out = spins > (1u << 24) || global_ns() - t0 > ex.wait_ns;
        if (out) atomicExch(ex.fault, 1u);
        if (__any_sync(0xffffffffu, out || *reinterpret_cast<volatile unsigned int*>(ex.fault) != 0u)) {
          if (lane == 0) sh.fault = 1;
          break;
        }
      }
    }
    // (a thread past the last block holds zeros)
    sh.packet[0][threadIdx.x] = __longlong_as_double((w[0] & 0xffffffffffffull) | (w[1] << 48));
    sh.packet[1][threadIdx.x] = __longlong_as_double(((w[1] >> 16) & 0xffffffffull) | (w[2] << 32));
    if (NV > 2) sh.packet[2][threadIdx.x] = __longlong_as_double(((w[2] >> 32) & 0xffffull) | (w[3] << 16));
  }
  __syncthreads();
  return warp < NV ? sum_strided(sh.packet[warp] + lane, (ex.count + 31) >> 5) : 0.0;
}

// the same for one value (FP64 or FP32) per thread and k; the first `warps` warps of the block
// hold values
template <bool RELEASE, int NV, class V, int T>
__device__ __forceinline__ double group_exchange(const ExchangeView& ex, unsigned int& epoch, const V (&v)[NV],
                                                 int warps, ExchangeShared<T>& sh) {
  if ((int)(threadIdx.x >> 5) < warps) {
#pragma unroll
    for (int k = 0; k < NV; ++k) reinterpret_cast<V*>(sh.part[k])[threadIdx.x] = v[k];
  }
  return exchange_stored<RELEASE, NV, V>(ex, epoch, warps, sh);
}

// the same for FP32 values, summed over a warp in FP32 (a few 1e-7, the precision of the vectors the products come
// from) and from there in FP64. The block may have more than T threads.
template <bool RELEASE, int NV, int T>
__device__ __forceinline__ double group_exchange_f32(const ExchangeView& ex, unsigned int& epoch, float (&v)[NV],
                                                     ExchangeShared<T>& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) sh.part[k][warp] = double(v[k]);
    if (warp == 0 && lane >= (int)(blockDim.x >> 5)) sh.part[k][lane] = 0.0;
  }
  return exchange_stored<RELEASE, NV, double>(ex, epoch, 1, sh);
}

// group_exchange for the blocks of one cluster (at most 16, the grid): the block sums go to the other blocks' shared
// memory, and the cluster's barrier, which releases the writes of all threads, is the only wait (the
// hardware's: the blocks of a cluster run together, and all take the same decisions from the same bits).
template <int NV, int T>
__device__ __forceinline__ double cluster_exchange(unsigned int& epoch, const double (&v)[NV], int warps,
                                                   ExchangeShared<T>& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  static_assert(3 * T >= 2 * 3 * 16, "two buffers");
  ++epoch;
  double* const remote = &sh.packet[0][0] + 16 * (3 * (epoch & 1) + warp);
  if (warp < warps) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sh.part[k][threadIdx.x] = v[k];
  }
  __syncthreads();
  if (warp < NV) {
    const double b = sum_strided(sh.part[warp] + lane, warps);
    const unsigned int here = static_cast<unsigned int>(__cvta_generic_to_shared(remote + blockIdx.x));
    unsigned int there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(min(lane, int(gridDim.x) - 1)));
    if (lane < (int)gridDim.x) asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(there), "d"(b) : "memory");
    __syncwarp();
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  double b = 0.0;
  if (warp < NV) {
    b = lane < (int)gridDim.x ? remote[lane] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    b = __shfl_sync(0xffffffffu, b, 0);
  }
  return b;
}

// The barrier alone, releasing the block's writes; thread 0 runs `meanwhile` between its arrival and its wait.
template <int T, class Meanwhile>
__device__ __forceinline__ void group_barrier(const ExchangeView& ex, unsigned int& epoch, ExchangeShared<T>& sh,
                                              Meanwhile meanwhile) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ++epoch;
  __syncthreads();
  if (ex.count == 1) {
    if (threadIdx.x == 0) meanwhile();
    __syncthreads();
    return;
  }
  unsigned long long* const base = ex.slots + (size_t)kSlot * (gridDim.x * (epoch & 1u) + ex.first);
  const unsigned long long tag = (unsigned long long)epoch << 48;
  if (threadIdx.x == 0) {
    fence_acq_rel_gpu();
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(base + kSlot * (blockIdx.x - ex.first)), "l"(tag) : "memory");
    meanwhile();
  }
  if (warp * 32 < ex.count) {
    unsigned long long w = 0, t0 = 0;
    bool wait = (int)threadIdx.x < ex.count;
    for (unsigned int spins = 1;; ++spins) {
      if (wait) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(base + kSlot * threadIdx.x) : "memory");
        wait = ((w ^ tag) >> 48) != 0;
      }
      if (!__any_sync(0xffffffffu, wait)) break;
      if (spins == 1u) t0 = global_ns();
      else if (spins == 2u || (spins & 255u) == 0u) {
        const bool out = spins > (1u << 24) || global_ns() - t0 > ex.wait_ns;
        if (out) atomicExch(ex.fault, 1u);
        if (__any_sync(0xffffffffu, out || *reinterpret_cast<volatile unsigned int*>(ex.fault) != 0u)) {
          if (lane == 0) sh.fault = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
}

}  // namespace gdt
