// Multi-right-hand-side EbE PCG: k load cases on one mesh (3D, edge-fan form).
//
// Node vectors hold all K cases of a node contiguously: [node][K][4] (K >= k,
// a power of two <= kMaxCases; unused cases stay zero). The matvec works on
// items (patch, chunk of C cases): the lanes of a warp hold C cases of 32 / C
// half-fans, so a node's values for the chunk are one contiguous C x 16-byte
// load, every gradient read from the patch block (kernels_fan_tma.cuh) is a
// broadcast serving C cases, and the forces go to the block's node-sorted
// force list ([entry][3][C]), whose runs the node sums add up without atomics. Every case has
// its own PCG scalars and stopping test; a converged case is frozen (its items
// are skipped once all C cases of a chunk are done).
#pragma once

#include "kernels.cuh"
#include "kernels_fan_tma.cuh"

namespace cfem {

constexpr int kMaxCases = 256;

// Scalars of a case. The two kernels of an iteration pass their per-case sums
// on as FP64 atomic additions and every CTA of the kernel behind derives what
// it needs from them (no last-block phase: its two levels of ticket, fences and
// serial FP64 additions took most of an iteration of few cases). A kernel reads
// only what the kernel before it wrote; CTA 0 publishes:
//   matvec of iteration `it` (parity q = it & 1): reads sum_b[q ^ 1], alpha,
//     inv_gamma, done[q ^ 1], ctl->iter; writes gamma, gamma_prev, beta, rr,
//     iters, done[q], ctl->all_done; empties sum_b[q]; adds p.Ap to sum_a[q];
//   vector kernel: reads sum_a[q], gamma, done[q], ctl->all_done; writes sigma,
//     alpha, inv_gamma, ctl->iter; empties sum_a[q ^ 1]; adds r.z, r.r to sum_b[q].
struct MultiScalars {
  double gamma, gamma_prev, gamma0, sigma, alpha, beta, rr, ff;
  double gamma_stop, rr_stop, inv_gamma;  // tol gamma0, (tol ||f||)^2, 1 / gamma
  double sum_a[2], sum_b[2][2];
  int done[2], iters;  // done: 0 running, 1 converged, 2 diverged, 3 iteration cap
  int pad;
};

struct MultiCtl {  // shared by the cases of one solve
  double tol;
  int rule, maxit, iter, all_done;
  int k_active;     // cases 0..k_active-1 are real, the rest are padding
  int loops;        // graph loop: bodies started in this run
  int loop_ok, pad;
};

template <typename T>
struct MultiParams {
  int n_patches;
  const int32_t *node_off, *own;
  const T *diagA;       // [node][4] diagonal of the operator (constrained DOFs)
  T lam, mu;
  int K;                // cases per node (power of two)
  int64_t n_nodes;
  MultiScalars *sc;     // [K]
  MultiCtl *ctl;
  int parity;           // of the iteration
  unsigned long long cond;  // iterations inside a graph loop (0: host loop), see k_pcg_update
  int cond_role, cond_chunk;
  FanTmaParams F;       // patch blocks (layout and fan offsets)
};

// Shared memory of k_matvec_multi<MODE, C> for K cases: the patch block, the
// staged node values [npn][C][4], per-case energies [K] and warp partials
// [8][C] (double), the mbarrier, the force list [kFanForces x kFanThreads][3][C],
// per-case beta and done flags [K].
struct MultiSmem {
  int sp, en, red, bar, fs, beta, done, bytes;
};
__host__ __device__ inline MultiSmem multi_smem(const FanBlockLayout &L, int C, int K) {
  MultiSmem m{};
  int off = L.bytes;
  m.sp = off; off += L.npn * C * 16;
  m.en = off; off += K * 8;
  m.red = off; off += (kHfanThreads / 32) * C * 8;
  m.bar = off; off += 16;
  m.fs = off; off += kFanForces * kFanThreads * 3 * C * 4;
  m.beta = off; off += K * 4;
  m.done = off; off += K * 4;
  m.bytes = off;
  return m;
}

// y_c += K' p_c for the K cases. PCG (MODE MV_PCG): p_c = z_c + beta_c p_old_c
// staged on the fly (written back by the owning patch), sigma_c = p_c.K'p_c.
// PLAIN: y_c += K' x_c. FP32 only (the patch blocks hold FP32 gradients).
//
// Items q = patch * (K / C) + chunk; CTA b takes the contiguous items
// [n b / G, n (b + 1) / G), so the chunks of a patch reuse its block. Lane l of
// warp w holds case l % C of half-fan (round * 8 + w) * (32 / C) + l / C: the
// two halves of a fan are lanes l and l ^ C. A thread's case (l % C) is the
// same in every phase, so its energy partial needs no exchange until the end
// of the item.
template <int MODE, int C>
__global__ void __launch_bounds__(kHfanThreads, C <= 2 ? 3 : 2) k_matvec_multi(MultiParams<float> P, const float *x,
                                                                  const float *pold, float *pnew, float *y) {
  using T = float;
  constexpr int DIM = 3, VW = 4, NW = kHfanThreads / 32;
  constexpr int HPW = 32 / C;                    // half-fans per warp and round
  constexpr int ROUNDS = kHfanThreads / (NW * HPW);
  constexpr int SU = C <= 2 ? 2 : 4;             // staging items in flight per thread
  static_assert(C == 2 || C == 4 || C == 8, "C: 2, 4 or 8 cases per item");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const FanBlockLayout &L = P.F.L;
  const int K = P.K, NC = K / C;
  const MultiSmem S = multi_smem(L, C, K);
  unsigned char *B = smem_raw;
  T *sp = reinterpret_cast<T *>(smem_raw + S.sp);
  double *s_en = reinterpret_cast<double *>(smem_raw + S.en);
  double *s_red = reinterpret_cast<double *>(smem_raw + S.red);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw + S.bar);
  T *fs = reinterpret_cast<T *>(smem_raw + S.fs);
  T *s_beta = reinterpret_cast<T *>(smem_raw + S.beta);
  int *s_done = reinterpret_cast<int *>(smem_raw + S.done);
  const int q = P.parity;
  for (int c = threadIdx.x; c < K; c += blockDim.x) {
    s_en[c] = 0;
    s_done[c] = 0;
    s_beta[c] = 0;
  }
  if (MODE == MV_PCG) {
    // every CTA: beta and the stopping tests from the update's sums (one thread
    // per case; K is at most the block size)
    bool stop = true;
    if (threadIdx.x < K) {
      const int c = threadIdx.x;
      MultiScalars &m = P.sc[c];
      const int it = P.ctl->iter;
      int done = m.done[q ^ 1];
      double b = 0;
      if (!done && it > 0) {
        const double g = m.sum_b[q ^ 1][0], rr = m.sum_b[q ^ 1][1];
        const int rule = P.ctl->rule;
        const double v = rule == 0 ? g : rr, limit = rule == 0 ? m.gamma_stop : m.rr_stop;
        if (!finite_bits(g) || !finite_bits(m.alpha)) done = 2;
        else if (rule == 0 ? v < limit : rule == 1 && v <= limit) done = 1;
        else if (it >= P.ctl->maxit) done = 3;
        b = g * m.inv_gamma;
        if (blockIdx.x == 0) {
          m.gamma_prev = m.gamma;
          m.gamma = g;
          m.rr = rr;
          m.beta = b;
          m.iters = it;
        }
      }
      if (blockIdx.x == 0) {
        m.done[q] = done;
        m.sum_b[q][0] = m.sum_b[q][1] = 0;
      }
      s_done[c] = done;
      s_beta[c] = done ? T(0) : (T)b;
      stop = done != 0;
    }
    const bool all = __syncthreads_and(stop);
    if (blockIdx.x == 0 && threadIdx.x == 0) P.ctl->all_done = all;
    if (all) return;
  }
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const uint16_t *fstart = reinterpret_cast<const uint16_t *>(B + L.fstart_off);
  const int32_t *nodes = reinterpret_cast<const int32_t *>(B + L.nodes_off);
  const uint8_t *bits = B + L.bits_off;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int cl = lane & (C - 1), hs = lane / C, h = hs & 1;
  const T lam = P.lam, mu = P.mu;
  const int64_t n_items = (int64_t)P.n_patches * NC;
  const int64_t q0 = n_items * blockIdx.x / gridDim.x, q1 = n_items * (blockIdx.x + 1) / gridDim.x;
  int cur = -1;
  unsigned nload = 0;
  for (int64_t item = q0; item < q1; ++item) {
    const int patch = (int)(item / NC), c0 = (int)(item - (int64_t)patch * NC) * C;
    if (MODE == MV_PCG) {
      bool all = true;  // (uniform: read from shared memory)
#pragma unroll
      for (int r = 0; r < C; ++r) all &= s_done[c0 + r] != 0;
      if (all) continue;
    }
    if (patch != cur) {
      fence_proxy_async();  // earlier reads of the block precede the copy that overwrites it
      __syncthreads();
      if (threadIdx.x == 0) {
        mbar_expect_tx(&bar[0], (unsigned)L.bytes);
        bulk_load(B, P.F.blocks + (size_t)patch * L.bytes, (unsigned)L.bytes, &bar[0]);
      }
      const bool ok = mbar_wait_bounded(&bar[0], nload & 1u);
      ++nload;
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) *(volatile int *)P.F.err = kErrTmaTimeout;
        return;
      }
      cur = patch;
    }
    const int32_t *hdr = reinterpret_cast<const int32_t *>(B + L.hdr_off);
    const int nn = hdr[0], own = hdr[1];
    const int n_it = nn * C;  // staging / output items (node i, case cl): it = i * C + cl
    const T beta = MODE == MV_PCG ? s_beta[c0 + cl] : T(0);
    const bool case_done = MODE == MV_PCG && s_done[c0 + cl] != 0;
    // 1. stage the chunk's node values: C cases of a node are one contiguous load
    for (int i0 = threadIdx.x; i0 < n_it; i0 += SU * kHfanThreads) {
      NodeV<T, VW> v[SU], w[SU];
      int gi[SU];
#pragma unroll
      for (int u = 0; u < SU; ++u) {
        const int it = i0 + u * kHfanThreads;
        gi[u] = it < n_it ? nodes[it / C] : -1;
        if (gi[u] >= 0) {
          const int64_t idx = (int64_t)gi[u] * K + c0 + cl;
          v[u] = ldv<T, VW>(x, idx);
          if (MODE == MV_PCG && beta != T(0)) w[u] = ldv<T, VW>(pold, idx);
        }
      }
#pragma unroll
      for (int u = 0; u < SU; ++u) {
        if (gi[u] < 0) continue;
        const int it = i0 + u * kHfanThreads, i = it / C;
        if (MODE == MV_PCG) {
          if (beta != T(0)) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) v[u].v[d] += beta * w[u].v[d];
          }
          // a stopped case keeps its last direction (a continued refinement
          // step starts from it); its lanes still compute, unused
          if (i >= own && !case_done) stv<T, VW>(pnew, (int64_t)gi[u] * K + c0 + cl, v[u]);
        }
        const unsigned bb = bits[i];
        NodeV<T, VW> m;
#pragma unroll
        for (int d = 0; d < VW; ++d) m.v[d] = (d < DIM && !(bb >> d & 1u)) ? v[u].v[d] : T(0);
        stv<T, VW>(sp, it, m);
      }
    }
    __syncthreads();
    // 2. half-fans: forces relative to P (missing tets have zero gradients),
    //    halves combined by shuffle, written to the force list
    Comp32 energy;
#pragma unroll 1
    for (int rd = 0; rd < ROUNDS; ++rd) {
      const int hf = (rd * NW + wid) * HPW + hs;
      int slot[6];
      const int nk = load_half_slots(B + L.slot_off, hf, slot);
      T du[6][DIM], fv[6][DIM];
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        NodeV<T, VW> s;
#pragma unroll
        for (int d = 0; d < VW; ++d) s.v[d] = 0;
        if (k < nk) s = ldv<T, VW>(sp, slot[k] * C + cl);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          du[k][d] = s.v[d];
          fv[k][d] = 0;
        }
      }
#pragma unroll
      for (int k = 1; k < 6; ++k)
#pragma unroll
        for (int d = 0; d < DIM; ++d) du[k][d] -= du[0][d];
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) {
        T G[9];
        load_tet_G(B + L.g_off, hf, jj, G);
        tet_forces_acc<T>(du[1], du[2 + jj], du[3 + jj], G, lam, mu, fv[1], fv[2 + jj], fv[3 + jj]);
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d) fv[0][d] = -(fv[1][d] + fv[2][d] + fv[3][d] + fv[4][d] + fv[5][d]);
      if (MODE == MV_PCG) {  // the forces sum to zero: sum_k u_k.f_k = sum_k>0 du_k.f_k
        T e = 0;
#pragma unroll
        for (int k = 1; k < 6; ++k)
#pragma unroll
          for (int d = 0; d < DIM; ++d) e += du[k][d] * fv[k][d];
        energy.add(e);
      }
      combine_half_forces<T, DIM, C>(fv, h);
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (k < nk && half_writes(h, k)) {
          T *o = fs + half_fpos(B + L.fpos_off, hf, k) * (3 * C) + cl;
#pragma unroll
          for (int d = 0; d < DIM; ++d) o[d * C] = fv[k][d];
        }
    }
    __syncthreads();
    // 3. node sums over contiguous force runs, constrained DOFs: (I - P) diag(A) p on owned nodes
    for (int it = threadIdx.x; it < n_it; it += kHfanThreads) {
      const int i = it / C;
      const unsigned bb = bits[i];
      T acc[DIM] = {0, 0, 0};
      const int k1 = fstart[i + 1];
      for (int k = fstart[i]; k < k1; ++k) {
        const T *f = fs + k * (3 * C) + cl;
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc[d] += f[d * C];
      }
      NodeV<T, VW> out;
      bool any = false;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        out.v[d] = (bb >> d & 1u) ? T(0) : acc[d];
        any |= out.v[d] != T(0);
      }
      out.v[3] = 0;
      const int g = nodes[i];
      const int64_t idx = (int64_t)g * K + c0 + cl;
      if ((bb & kBcBits) && i >= own) {
        const NodeV<T, VW> v = ldv<T, VW>(MODE == MV_PCG ? pnew : x, idx);  // this block wrote pnew[idx] while staging
        const NodeV<T, VW> dg = ldv<T, VW>(P.diagA, g);
#pragma unroll
        for (int d = 0; d < DIM; ++d)
          if (bb >> d & 1u) {
            const T t = dg.v[d] * v.v[d];
            out.v[d] = t;
            any |= t != T(0);
            if (MODE == MV_PCG) energy.add(t * v.v[d]);
          }
      }
      if (any) atomic_addv<T, VW>(y, idx, out, DIM);
    }
    if (MODE == MV_PCG) {  // per-case energy of the item: lanes of one case, then warps in order
#pragma unroll
      for (int o = C; o < 32; o <<= 1) {
        const float h2 = __shfl_xor_sync(0xffffffffu, energy.hi, o), l2 = __shfl_xor_sync(0xffffffffu, energy.lo, o);
        energy.merge(h2, l2);
      }
      if (lane < C) s_red[wid * C + lane] = (double)energy.hi + (double)energy.lo;
    }
    __syncthreads();  // sp, fs and s_red of this item are complete
    if (MODE == MV_PCG && threadIdx.x < 8 * C) {  // (a tree of eight lanes per case)
      double t = s_red[(threadIdx.x & 7) * C + (threadIdx.x >> 3)];
      const unsigned mask = C < 4 ? (1u << (8 * (C & 3))) - 1u : 0xffffffffu;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(mask, t, o);
      if ((threadIdx.x & 7) == 0) s_en[c0 + (threadIdx.x >> 3)] += t;
    }
  }
  if (MODE != MV_PCG) return;
  __syncthreads();
  for (int c = threadIdx.x; c < K; c += blockDim.x)
    if (!s_done[c]) atomicAdd(&P.sc[c].sum_a[q], s_en[c]);
}

// z_c += beta_c p_c for every (node, case) item, p_c read from pB when
// parity_c is 0, from pA when 1 (cases with beta_c = 0 are left alone): the
// first direction of a continued multi-RHS run.
static __global__ void k_multi_fold(int64_t n_items, int K, const float *beta, const int *parity, const float *pA,
                                    const float *pB, float *z) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= n_items) return;
  const int c = (int)(q % K);
  const float b = beta[c];
  if (b == 0.f) return;
  const NodeV<float, 4> p = ldv<float, 4>(parity[c] ? pA : pB, q);
  NodeV<float, 4> v = ldv<float, 4>(z, q);
#pragma unroll
  for (int d = 0; d < 3; ++d) v.v[d] += b * p.v[d];
  stv<float, 4>(z, q, v);
}

// Per case: init (r = f, x = 0; sums r.z, r.r, f.f into sum_b[0], sum_a[0]) or
// update (x += alpha p, r -= alpha u; sums r.z, r.r), z = M^-1 r, u = 0. Items
// are (node, case) with the case fastest; the grid stride is a multiple of K, so
// a thread always works on the same case.
// LOOP: the instance for the graph loop; its condition is driven like
// k_pcg_update's.
template <typename T, bool LOOP = false>
__global__ void __launch_bounds__(kThreads) k_pcg_multi_vec(MultiParams<T> P, T *xv, T *r, T *z, const T *p, T *u,
                                                           const T *f, const T *dinv, int init) {
  constexpr int DIM = 3, VW = 4;
  const int K = P.K, q = P.parity;
  // the case scalars once per CTA (one thread per case), the shared flag by
  // thread 0: every thread reading the same lines would queue at one L2 slice
  __shared__ T s_alpha[kMaxCases];
  __shared__ int s_frozen[kMaxCases], s_all;
  if (threadIdx.x == 0) {
    s_all = init ? 0 : P.ctl->all_done;
    if constexpr (LOOP)
      if (blockIdx.x == 0) {
        if (P.cond_role & 1) {
          const int nl = ++P.ctl->loops;
          P.ctl->loop_ok = nl <= P.ctl->maxit / P.cond_chunk + 16;
          cudaGraphSetConditional(P.cond, 0u);
        }
        if (P.cond_role & 2) cudaGraphSetConditional(P.cond, !s_all && P.ctl->loop_ok ? 1u : 0u);
      }
  }
  for (int cc = threadIdx.x; cc < K; cc += blockDim.x) {
    MultiScalars &m = P.sc[cc];
    const int fz = !init && m.done[q];
    double alpha = 0;
    if (!init && !fz) {
      const double sigma = m.sum_a[q];
      alpha = m.gamma / sigma;
      if (blockIdx.x == 0) {
        m.sigma = sigma;
        m.alpha = alpha;
        m.inv_gamma = 1.0 / m.gamma;
      }
    }
    if (!init && blockIdx.x == 0) m.sum_a[q ^ 1] = 0;
    s_frozen[cc] = fz;
    s_alpha[cc] = (T)alpha;
  }
  if (!init && blockIdx.x == 0 && threadIdx.x == 0) P.ctl->iter += 1;
  __syncthreads();
  if (s_all) return;
  const int c = threadIdx.x & (K - 1);
  const bool frozen = s_frozen[c] != 0;
  const T alpha = s_alpha[c];
  DotAcc<T> acc[3];  // r.z, r.r, f.f
  const int64_t n_items = P.n_nodes * K;
  // U items per thread per round, all loads issued before any is used; the
  // stride is a multiple of K, so every item of a thread is case c
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n_items; i0 += stride * U) {
    NodeV<T, VW> zero;
#pragma unroll
    for (int d = 0; d < VW; ++d) zero.v[d] = 0;
    if (frozen) {
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (i0 + k * stride < n_items) stv<T, VW>(u, i0 + k * stride, zero);
      continue;
    }
    NodeV<T, VW> di[U], rv[U], xx[U], pp[U], uu[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int64_t i = i0 + k * stride;
      if (i >= n_items) continue;
      di[k] = ldv<T, VW>(dinv, i / K);
      if (init) {
        rv[k] = ldv<T, VW>(f, i);
      } else {
        rv[k] = ldv<T, VW>(r, i);
        xx[k] = ldv<T, VW>(xv, i);
        pp[k] = ldv<T, VW>(p, i);
        uu[k] = ldv<T, VW>(u, i);
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int64_t i = i0 + k * stride;
      if (i >= n_items) continue;
      NodeV<T, VW> zz = zero;
      if (init) {
        xx[k] = zero;
      } else {
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          xx[k].v[d] += alpha * pp[k].v[d];
          rv[k].v[d] -= alpha * uu[k].v[d];
        }
      }
      T rz = 0, rr = 0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        zz.v[d] = rv[k].v[d] * di[k].v[d];
        rz += rv[k].v[d] * zz.v[d];
        rr += rv[k].v[d] * rv[k].v[d];
      }
      acc[0].add(rz);
      acc[1].add(rr);
      if (init) acc[2].add(rr);
      stv<T, VW>(xv, i, xx[k]);
      stv<T, VW>(r, i, rv[k]);
      stv<T, VW>(z, i, zz);
      stv<T, VW>(u, i, zero);
    }
  }
  // Totals of the block per case: lanes of the same case merge as compensated
  // FP32, the warps' sums add up in FP64, one atomic addition per case and sum.
  constexpr int NW = kThreads / 32;
  __shared__ double red[3][NW * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, KW = min(K, 32);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k == 2 && !init) break;
    Comp32 a = acc[k].c;
    for (int o = 16; o >= KW; o >>= 1) {
      const float h2 = __shfl_xor_sync(0xffffffffu, a.hi, o), l2 = __shfl_xor_sync(0xffffffffu, a.lo, o);
      a.merge(h2, l2);
    }
    if (lane < KW) red[k][wid * 32 + lane] = (double)a.hi + (double)a.lo;
  }
  __syncthreads();
  // warps w, w + K / 32, ... hold case (w mod (K / 32)) 32 + lane
  const int groups = K / KW, n_sums = init ? 3 : 2;
  for (int t = threadIdx.x; t < K * n_sums; t += blockDim.x) {
    const int cc = t & (K - 1), k = t / K;
    if (s_frozen[cc]) continue;
    double v = 0;
    for (int w = cc / KW; w < NW; w += groups) v += red[k][w * 32 + (cc & (KW - 1))];
    MultiScalars &m = P.sc[cc];
    atomicAdd(k == 2 ? &m.sum_a[0] : &m.sum_b[init ? 0 : q][k], v);
  }
}

// After the init kernel: the scalars of every case (one block).
static __global__ void __launch_bounds__(kMaxCases) k_multi_start(MultiScalars *sc, MultiCtl *ctl, int K) {
  const int c = threadIdx.x;
  bool stop = true;
  if (c < K) {
    MultiScalars &m = sc[c];
    const double g = m.sum_b[0][0], rr = m.sum_b[0][1], ff = m.sum_a[0], lim = ctl->tol * sqrt(ff);
    m.gamma0 = m.gamma = m.gamma_prev = g;
    m.rr = rr;
    m.ff = ff;
    m.gamma_stop = ctl->tol * g;
    m.rr_stop = lim < 0 ? -1.0 : lim * lim;  // (a negative tol stops nothing)
    m.iters = 0;
    m.sigma = m.alpha = m.beta = 0;
    m.inv_gamma = 0;
    m.sum_a[0] = m.sum_a[1] = 0;
    int done = 0;
    if (c >= ctl->k_active || g == 0.0) done = 1;
    else if (ctl->rule == 1 && rr <= m.rr_stop) done = 1;
    else if (!isfinite(g)) done = 2;
    m.done[0] = m.done[1] = done;
    stop = done != 0;
  }
  const bool all = __syncthreads_and(stop);
  if (c == 0) {
    ctl->iter = 0;
    ctl->all_done = all;
  }
}

// caller order F[c][n_dof] (FP64) -> dst[node][K][4] (T), scaled; cases >= k zero
template <typename T>
__global__ void k_multi_to_internal(int64_t nn, int K, int k, int64_t nd, const double *F, const int32_t *new2old,
                                    T *dst) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nn * K) return;
  const int64_t n = q / K;
  const int c = (int)(q - n * K);
  const int64_t o = new2old[n];
  NodeV<T, 4> v;
#pragma unroll
  for (int d = 0; d < 4; ++d) v.v[d] = (c < k && d < 3) ? (T)F[(size_t)c * nd + o * 3 + d] : T(0);
  stv<T, 4>(dst, q, v);
}

template <typename T>
__global__ void k_multi_to_caller(int64_t nn, int K, int k, int64_t nd, const T *src, const int32_t *new2old,
                                  double *U) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nn * K) return;
  const int64_t n = q / K;
  const int c = (int)(q - n * K);
  if (c >= k) return;
  const int64_t o = new2old[n];
  const NodeV<T, 4> v = ldv<T, 4>(src, q);
#pragma unroll
  for (int d = 0; d < 3; ++d) U[(size_t)c * nd + o * 3 + d] = (double)v.v[d];
}

// x64 += d32 over whole multi arrays
static __global__ void k_multi_accumulate(int64_t n, const float *d, double *x) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) x[i] += (double)d[i];
}

}  // namespace cfem
