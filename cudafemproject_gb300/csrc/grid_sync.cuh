// Grid-wide sums and barriers inside a cooperative kernel (all CTAs resident).
//
// A sum: every CTA publishes its partial in a slot of its own and every CTA
// adds all slots up itself, in CTA order, so that all hold bit-identical totals
// and no second pass or broadcast is needed: one trip through L2 is the barrier
// and the reduction. A slot holds kSlotEmpty until its CTA has published. A
// loop that alternates sums and barriers uses two sets of slots in turn: those
// of the next iteration are emptied (grid_reset) once a sum of this iteration
// has shown that every CTA has left the last one, and the barrier that ends
// this iteration orders that before their next use.
//
// Every slot exists in one copy per kGridReaders CTAs: polls of one line queue
// at its L2 slice (152 CTAs polling the same flags took 5.8 us, with 19 copies
// 1.8 us; a barrier on one atomic counter, one poller per CTA, takes 1.4 us, 2.2
// with its two fences).
//
// One FP64 instruction of a warp holds its quarter of the SM for 64 cycles on
// GB300, whatever lanes take part (measured: 64.5 cycles with 1, 8, 16 or 32
// active lanes; 16 warps doing the same chain take 259). So the partials of a
// block go through shared memory to four warps, one per quarter, instead of a
// shuffle tree in every warp, and divisions are done by one warp only.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cfem {

constexpr int kMaxGridSums = 3;  // sums per exchange
constexpr int kGridReaders = 8;
constexpr unsigned long long kSlotEmpty = ~0ull;  // (a NaN pattern; sums that are NaN are stored as another one)

struct GridSync {
  unsigned long long *slots;  // [sets][kMaxGridSums][copies][grid], all kSlotEmpty at launch
  unsigned *arrived;          // CTAs arrived at barriers, zero at launch
  long long limit;            // clock64 cycles a CTA waits for the others
  int absent_plus1;           // self-test: CTA that leaves the kernel at its start, plus one; else 0
};

__host__ __device__ inline int grid_copies(int grid) { return (grid + kGridReaders - 1) / kGridReaders; }
inline size_t grid_slots_count(int sets, int grid) { return (size_t)sets * kMaxGridSums * grid_copies(grid) * grid; }

template <int THREADS>
struct GridShared {
  double part[kMaxGridSums][THREADS];
  double quarter[kMaxGridSums][4];
  double total[kMaxGridSums + 2];  // totals, then what `then` leaves for the block
  int ok;
};

__device__ __forceinline__ unsigned long long slot_load(const unsigned long long *p) {
  unsigned long long u;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
  return u;
}
__device__ __forceinline__ void slot_store(unsigned long long *p, unsigned long long u) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}

// v[k]: sum over all threads of the grid (set: which slots; all threads call).
// `then(total)` runs in warp 0 between the totals and the block's barrier (its
// lanes all hold them) and may leave results in sh.total[kMaxGridSums ..].
// This orders no other memory. False if some CTA did not arrive within the
// limit: the caller leaves the kernel without another exchange.
template <int N, int THREADS, typename F>
__device__ __forceinline__ bool grid_sums(const GridSync &G, int set, double (&v)[N], GridShared<THREADS> &sh, F then) {
  static_assert(N <= kMaxGridSums && THREADS % 128 == 0, "");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) sh.part[k][threadIdx.x] = v[k];
  __syncthreads();
  if (wid < 4) {
    double t[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      t[k] = sh.part[k][threadIdx.x];
#pragma unroll
      for (int q = 1; q < THREADS / 128; ++q) t[k] += sh.part[k][threadIdx.x + 128 * q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < N; ++k) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < N; ++k) sh.quarter[k][wid] = t[k];
  }
  __syncthreads();
  if (wid == 0) {
    const int grid = gridDim.x, copies = grid_copies(grid);
    unsigned long long *now = G.slots + (size_t)set * kMaxGridSums * copies * grid;
    {
      unsigned long long mine[N];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const double t = (sh.quarter[k][0] + sh.quarter[k][1]) + (sh.quarter[k][2] + sh.quarter[k][3]);
        mine[k] = t != t ? 0x7FF8000000000000ull : (unsigned long long)__double_as_longlong(t);
      }
      for (int c = lane; c < copies; c += 32)
#pragma unroll
        for (int k = 0; k < N; ++k) slot_store(now + ((size_t)k * copies + c) * grid + blockIdx.x, mine[k]);
    }
    now += (size_t)(blockIdx.x / kGridReaders) * grid;
    const long long t0 = clock64();
    double s[N];
    bool ok = true;
    for (int b0 = 0; b0 < grid; b0 += 160) {  // five slots per lane and sum in flight
      unsigned long long u[N][5];
      for (;;) {
        bool all = true;
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const int b = b0 + q * 32 + lane;
            u[k][q] = b < grid ? slot_load(now + (size_t)k * copies * grid + b) : 0ull;
          }
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int k = 0; k < N; ++k) all &= u[k][q] != kSlotEmpty;
        ok = __all_sync(0xffffffffu, all);
        if (ok || clock64() - t0 > G.limit) break;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        double w[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = __longlong_as_double((long long)u[k][q]);
        const double t = ((w[0] + w[1]) + (w[2] + w[3])) + w[4];
        s[k] = b0 ? s[k] + t : t;
      }
    }
    if (ok) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < N; ++k) sh.total[k] = s[k];
      then(s);
    }
    if (lane == 0) sh.ok = ok;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = sh.total[k];
  return sh.ok != 0;
}

// Empties this CTA's slots of the first N sums of a set.
template <int N>
__device__ __forceinline__ void grid_reset(const GridSync &G, int set) {
  const int copies = grid_copies(gridDim.x);
  for (int t = threadIdx.x; t < N * copies; t += blockDim.x)
    slot_store(G.slots + ((size_t)set * kMaxGridSums * copies + t) * gridDim.x + blockIdx.x, kSlotEmpty);
}

// Grid barrier: every global write before it is seen by every plain read
// after it. epoch: 1, 2, 3, ... False on a timeout.
template <int THREADS>
__device__ __forceinline__ bool grid_barrier(const GridSync &G, unsigned epoch, GridShared<THREADS> &sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = epoch * gridDim.x;  // (compared modulo 2^32)
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(G.arrived) : "memory");
    const long long t0 = clock64();
    bool ok = true;
    for (;;) {
      unsigned v;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(G.arrived) : "memory");
      if ((int)(v - target) >= 0) break;
      if (clock64() - t0 > G.limit) {
        ok = false;
        break;
      }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    sh.ok = ok;
  }
  __syncthreads();
  return sh.ok != 0;
}

}  // namespace cfem
