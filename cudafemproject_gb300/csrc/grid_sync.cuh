// Grid-wide sums inside a cooperative kernel (all CTAs resident).
//
// Every CTA publishes its partial sums in slots of its own and every CTA adds
// all slots up itself, in CTA order, so that all of them hold bit-identical
// totals and no second pass or broadcast is needed: one round trip through L2
// is the barrier and the reduction. A slot holds the sentinel until its CTA
// has published. Three sets of slots take turns: a CTA that publishes in
// exchange k has seen every CTA publish in exchange k - 1, hence every CTA has
// finished reading exchange k - 2, whose set (k + 1) mod 3 it resets for the
// next exchange before it publishes.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cfem {

constexpr int kMaxGridSums = 3;   // sums per exchange
constexpr int kGridSyncWarps = 32;
constexpr unsigned long long kSlotEmpty = ~0ull;  // (a NaN pattern; sums that are NaN are stored as another one)

inline size_t grid_slots_bytes(int grid) { return (size_t)3 * kMaxGridSums * grid * sizeof(double); }

struct GridSync {
  unsigned long long *slots;  // [3][kMaxGridSums][grid], all kSlotEmpty at launch
  long long limit;            // clock64 cycles a CTA waits for the others
  unsigned exchange;          // of this thread (the same everywhere)
};

struct GridShared {
  double part[kMaxGridSums][kGridSyncWarps];
  double total[kMaxGridSums];
  int ok;
};

// Adds v over all threads of the grid (all threads call; v holds the totals
// afterwards) and orders every global write before it against every read
// after it. False if some CTA did not arrive within the limit: the caller
// returns from the kernel without another exchange.
template <int N>
__device__ __forceinline__ bool grid_sums(GridSync &G, double (&v)[N], GridShared &sh) {
  static_assert(N <= kMaxGridSums, "");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) sh.part[k][wid] = v[k];
  }
  __syncthreads();
  if (wid == 0) {
    const int grid = gridDim.x, nw = blockDim.x >> 5;
    unsigned long long *now = G.slots + (size_t)(G.exchange % 3) * kMaxGridSums * grid;
    unsigned long long *next = G.slots + (size_t)((G.exchange + 1) % 3) * kMaxGridSums * grid;
    double s[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double t = lane < nw ? sh.part[k][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      s[k] = t;
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < kMaxGridSums; ++k)
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(next + k * grid + blockIdx.x), "l"(kSlotEmpty) : "memory");
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const unsigned long long bits =
            s[k] != s[k] ? 0x7FF8000000000000ull : (unsigned long long)__double_as_longlong(s[k]);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(now + k * grid + blockIdx.x), "l"(bits) : "memory");
      }
    }
    const long long t0 = clock64();
    bool ok;
    for (;;) {
      bool all = true;
#pragma unroll
      for (int k = 0; k < N; ++k) s[k] = 0;
      for (int b0 = 0; b0 < grid; b0 += 160) {  // five loads in flight per sum and lane
        unsigned long long u[N][5];
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const int b = b0 + q * 32 + lane;
            u[k][q] = 0;
            if (b < grid)
              asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u[k][q]) : "l"(now + k * grid + b) : "memory");
          }
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int k = 0; k < N; ++k) {
            all &= u[k][q] != kSlotEmpty;
            s[k] += __longlong_as_double((long long)u[k][q]);
          }
      }
      ok = __all_sync(0xffffffffu, all);
      if (ok || clock64() - t0 > G.limit) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
    for (int k = 0; k < N; ++k) {
      for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      if (lane == 0) sh.total[k] = s[k];
    }
    if (lane == 0) sh.ok = ok;
  }
  __syncthreads();
  ++G.exchange;
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = sh.total[k];
  return sh.ok != 0;
}

}  // namespace cfem
