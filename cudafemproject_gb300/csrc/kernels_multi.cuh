// Multi-right-hand-side EbE PCG: k load cases on one mesh (3D, edge-fan form).
//
// Node vectors hold all K cases of a node contiguously: [node][K][4] (K >= k,
// a power of two <= kMaxCases; unused cases stay zero). The matvec works on
// items (patch, chunk of C cases): a thread holds two cases of a half-fan, so a
// node's values for the chunk are one contiguous C x 16-byte load, every
// gradient read from the patch block (kernels_fan_tma.cuh) is a broadcast
// serving C cases, and the forces go to the block's node-sorted force list,
// whose runs the node sums add up without atomics. Every case has its own PCG
// scalars and stopping test; a converged case is frozen (its items are skipped
// once all C cases of a chunk are done).
#pragma once

#include "kernels.cuh"
#include "kernels_fan_tma.cuh"

namespace cfem {

constexpr int kMaxCases = 256;
constexpr int kReached = 5;
// A case that runs on with the others stops at this part of its (squared) limit,
// an order below the tolerance in the norm: where the FP32 recurrence is still
// the true residual.
constexpr double kReachedFloor = 1e-2;
__host__ __device__ inline bool case_stopped(int done) { return done != 0 && done != kReached; }

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
  // done: 0 running, 1 converged, 2 diverged, 3 iteration cap, 4 stopped by the
  // others, kReached: the test has been met, running on with the others (a norm
  // may rise again: at the end of the round it counts as it is then)
  int done[2], iters;
  int cap;  // iterations of this run at most
};

struct MultiCtl {  // shared by the cases of one solve
  double tol;
  int rule, maxit, iter, all_done;
  int k_active;     // cases 0..k_active-1 are real, the rest are padding
  int loops;        // graph loop: bodies started in this run
  int loop_ok;
  int quorum;       // cases that meet the test or are stopped (padding included) at which all stop, see MultiCont
};

// Offsets into the shared memory of k_matvec_multi (multi_smem), formed on the
// host: the kernel has no registers to spare for them.
struct MultiSmem {
  int tab, sp, en, red, bar, fs, beta, done, bytes;
};

template <typename T>
struct MultiParams {
  MultiSmem S;
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

// Two planes of shared memory for vectors of case pairs: (x0 x1 y0 y1) and (z0 z1).
struct PairPlanes {
  float4 *a;
  float2 *b;
  __device__ __forceinline__ PairPlanes(unsigned char *base, int n)
      : a(reinterpret_cast<float4 *>(base)), b(reinterpret_cast<float2 *>(base + (size_t)n * 16)) {}
  __device__ __forceinline__ void load(int i, float2 (&v)[3]) const {
    const float4 q = a[i];
    v[0] = make_float2(q.x, q.y);
    v[1] = make_float2(q.z, q.w);
    v[2] = b[i];
  }
  __device__ __forceinline__ void store(int i, const float2 (&v)[3]) const {
    a[i] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
    b[i] = v[2];
  }
};
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// tet_forces_acc for two cases at once: the same products and sums in the same
// order, each a packed FP32 instruction.
__device__ __forceinline__ void tet_forces_acc2(const float2 (&d1)[3], const float2 (&d2)[3], const float2 (&d3)[3],
                                                const float (&G)[9], float lam, float mu, float2 (&f1)[3],
                                                float2 (&f2)[3], float2 (&f3)[3]) {
  float2 H[3][3], g[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) g[k] = dup2(G[k]);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      H[i][j] = __ffma2_rn(d3[i], g[6 + j], __ffma2_rn(d2[i], g[3 + j], __fmul2_rn(d1[i], g[j])));
  const float2 l2 = dup2(lam), m2 = dup2(mu), mm2 = dup2(mu + mu);
  const float2 tr = __fmul2_rn(l2, __fadd2_rn(__fadd2_rn(H[0][0], H[1][1]), H[2][2]));
  float2 S[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i) S[i][i] = __ffma2_rn(mm2, H[i][i], tr);
  S[0][1] = S[1][0] = __fmul2_rn(m2, __fadd2_rn(H[0][1], H[1][0]));
  S[0][2] = S[2][0] = __fmul2_rn(m2, __fadd2_rn(H[0][2], H[2][0]));
  S[1][2] = S[2][1] = __fmul2_rn(m2, __fadd2_rn(H[1][2], H[2][1]));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    f1[i] = __ffma2_rn(S[i][2], g[2], __ffma2_rn(S[i][1], g[1], __ffma2_rn(S[i][0], g[0], f1[i])));
    f2[i] = __ffma2_rn(S[i][2], g[5], __ffma2_rn(S[i][1], g[4], __ffma2_rn(S[i][0], g[3], f2[i])));
    f3[i] = __ffma2_rn(S[i][2], g[8], __ffma2_rn(S[i][1], g[7], __ffma2_rn(S[i][0], g[6], f3[i])));
  }
}

// Threads of a CTA of k_matvec_multi<C>: 16 warps per SM in either case (the
// shared memory of 8 cases leaves one CTA per SM, that of 2 or 4 cases two).
// 8 cases in 256 threads: 172 us per iteration of 32 cases of 331,776 tets, in
// 512: 151 (then the fastest width; 4 cases: 171).
__host__ __device__ constexpr int multi_threads(int C) { return C == 8 ? 512 : 256; }

// Shared memory of k_matvec_multi<C> for K cases: the patch block, a second copy
// of its header and node tables (fstart, nodes, bits), the staged node values
// [npn][C / 2] (planes), per-case energies [K] and warp partials [warps][C]
// (compensated pairs), the mbarrier, the force list
// [kFanForces x kFanThreads][C / 2] (planes), per-case beta and done flags [K].
inline MultiSmem multi_smem(const FanBlockLayout &L, int C, int K) {
  MultiSmem m{};
  int off = L.bytes;
  m.tab = off; off += 16 + L.g_off - L.fstart_off;
  m.sp = off; off += L.npn * (C / 2) * 24;
  m.en = off; off += K * 8;
  m.red = off; off += (multi_threads(C) / 32) * C * 8;
  m.bar = off; off += 16;
  m.fs = off; off += kFanForces * kFanThreads * 3 * C * 4;
  m.beta = off; off += K * 4;
  m.done = off; off += K * 4;
  m.bytes = off;
  return m;
}

// u_c += K' p_c for the K cases, p_c = z_c + beta_c p_old_c staged on the fly
// (written back by the owning patch), sigma_c = p_c.K'p_c; FP32 (the patch
// blocks hold FP32 gradients).
//
// Items q = patch * (K / C) + chunk; CTA b takes the contiguous items
// [n b / G, n (b + 1) / G), so the chunks of a patch reuse its block. A thread
// works on two cases with packed FP32 instructions: lane l of warp w holds
// cases 2 (l % CL), 2 (l % CL) + 1 (CL = C / 2) of half-fan
// (round * warps + w) * (32 / CL) + l / CL; the two halves of a fan are lanes l
// and l ^ CL. A thread's cases are the same in every phase, so its energy
// partials need no exchange until the end of the item.
//
// Bound by the phases of an item (staging, half-fans, node sums) behind one
// another with 16 warps per SM; issue slots are 38% used, the L1 48%. Two cases
// per thread cut the instructions of a launch for 32 cases of 98,304 tets from
// 21.9 M to 14.0 M (of warps). One iteration, before and after: 32 cases of 98,304
// tets 52.0 -> 46.2 us, 8 cases 19.7 -> 16.4, 4 cases 14.4 -> 12.7; 32 cases of
// 331,776 tets 176 -> 148, 8 cases 43.8 -> 37.3. The registers are at their
// limit: forms that spill 50 bytes or more lost all of it (the next chunk's
// node values prefetched into registers, z formed here from r, the step to x
// taken here).
template <int C>
__global__ void __launch_bounds__(multi_threads(C), 512 / multi_threads(C))
    k_matvec_multi(MultiParams<float> P, const float *z, const float *pold, float *pnew, float *y) {
  using T = float;
  constexpr int DIM = 3, VW = 4, NT = multi_threads(C), NW = NT / 32;
  constexpr int CL = C / 2;                      // lanes per half-fan
  constexpr int HPW = 32 / CL;                   // half-fans per warp and round
  constexpr int ROUNDS = kHfanThreads / (NW * HPW);  // (256 half-fans of a patch)
  static_assert(C == 2 || C == 4 || C == 8, "C: 2, 4 or 8 cases per item");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const FanBlockLayout &L = P.F.L;
  const int K = P.K, NC = K / C;
  const MultiSmem &S = P.S;
  unsigned char *B = smem_raw;
  const PairPlanes sp(smem_raw + S.sp, L.npn * CL);
  double *s_en = reinterpret_cast<double *>(smem_raw + S.en);
  float2 *s_red = reinterpret_cast<float2 *>(smem_raw + S.red);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw + S.bar);
  const PairPlanes fs(smem_raw + S.fs, kFanForces * kFanThreads * CL);
  T *s_beta = reinterpret_cast<T *>(smem_raw + S.beta);
  int *s_done = reinterpret_cast<int *>(smem_raw + S.done);
  const int q = P.parity;
  for (int c = threadIdx.x; c < K; c += blockDim.x) {
    s_en[c] = 0;
    s_done[c] = 0;
    s_beta[c] = 0;
  }
  const int64_t n_items = (int64_t)P.n_patches * NC;  // (an int: the items of a mesh that fits the memory)
  const int q0 = (int)(n_items * blockIdx.x / gridDim.x), q1 = (int)(n_items * (blockIdx.x + 1) / gridDim.x);
  // the first patch's block (static operator data) is on its way before the
  // wait for the kernel before this one
  // Block of patch p, the header and node tables into copy t.
  auto issue_copy = [&](int p, int t) {
    const unsigned char *src = P.F.blocks + (size_t)p * L.bytes;
    mbar_expect_tx(&bar[0], (unsigned)L.bytes);
    if (t == 0) {
      bulk_load(B, src, (unsigned)L.bytes, &bar[0]);
    } else {
      bulk_load(smem_raw + S.tab, src, 16u, &bar[0]);
      bulk_load(smem_raw + S.tab + 16, src + L.fstart_off, (unsigned)(L.g_off - L.fstart_off), &bar[0]);
      bulk_load(B + L.slot_off, src + L.slot_off, (unsigned)(L.fstart_off - L.slot_off), &bar[0]);
      bulk_load(B + L.g_off, src + L.g_off, (unsigned)(L.bytes - L.g_off), &bar[0]);
    }
  };
  int coming = -1;  // patch whose copy has been issued and not waited for
  unsigned nload = 0;
  if (q0 < q1) {
    coming = q0 / NC;
    if (threadIdx.x == 0) {
      mbar_init(&bar[0], 1);
      fence_mbar_init();
      issue_copy(coming, 0);
    }
  }
  griddep_wait();
  // every CTA: beta and the stopping tests from the update's sums (one thread
  // per case; K is at most the block size)
  int done = 0;
  bool met = false;  // the test, in this iteration
  double b = 0;
  if (threadIdx.x < K) {
    const int c = threadIdx.x;
    MultiScalars &m = P.sc[c];
    const int it = P.ctl->iter;
    done = m.done[q ^ 1];
    if (!case_stopped(done) && it > 0) {
      const double g = m.sum_b[q ^ 1][0], rr = m.sum_b[q ^ 1][1];
      const int rule = P.ctl->rule;
      const double v = rule == 0 ? g : rr, limit = rule == 0 ? m.gamma_stop : m.rr_stop;
      if (!finite_bits(g) || !finite_bits(m.alpha)) done = 2;
      else if ((met = rule == 0 ? v < limit : rule == 1 && v <= limit))
        done = P.ctl->quorum <= K && v > kReachedFloor * limit ? kReached : 1;
      else if (it >= m.cap) done = 3;
      b = g * m.inv_gamma;
      if (blockIdx.x == 0) {
        m.gamma_prev = m.gamma;
        m.gamma = g;
        m.rr = rr;
        m.beta = b;
        m.iters = it;
      }
    }
  }
  const int n_done = __syncthreads_count(done != 0);
  if (threadIdx.x < K) {
    const int c = threadIdx.x;
    if (n_done >= P.ctl->quorum && P.ctl->iter > 0 && !case_stopped(done)) done = met ? 1 : 4;
    if (blockIdx.x == 0) {
      P.sc[c].done[q] = done;
      P.sc[c].sum_b[q][0] = P.sc[c].sum_b[q][1] = 0;
    }
    s_done[c] = case_stopped(done);
    s_beta[c] = case_stopped(done) ? T(0) : (T)b;
  }
  const bool all = __syncthreads_and(threadIdx.x >= K || case_stopped(done));
  if (blockIdx.x == 0 && threadIdx.x == 0) P.ctl->all_done = all;
  if (all) {
    if (threadIdx.x == 0 && coming >= 0) mbar_wait_bounded(&bar[0], 0u);  // (the copy lands before the CTA exits)
    return;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int cl = lane & (CL - 1), hs = lane / CL, h = hs & 1;
  const T lam = P.lam, mu = P.mu;
  // next item from i on with a case still running (uniform: from shared memory)
  auto next_live = [&](int i) {
    for (; i < q1; ++i) {
      const int c0 = i % NC * C;
      bool all = true;
#pragma unroll
      for (int r = 0; r < C; ++r) all &= s_done[c0 + r] != 0;
      if (!all) break;
    }
    return i;
  };
  int cur = -1, tab = 1;
  // node tables of the current patch, in copy `tab`
  auto table = [&](int off) { return smem_raw + (tab ? S.tab + 16 - L.fstart_off : 0) + off; };
  auto node = [&](int i) { return reinterpret_cast<const int32_t *>(table(L.nodes_off))[i]; };
  for (int item = next_live(q0), next; item < q1; item = next) {
    next = next_live(item + 1);
    if (next >= q1) griddep_launch_dependents();
    const int patch = item / NC, c0 = (item - patch * NC) * C;
    if (patch != cur) {
      bool ok = true;
      tab ^= 1;
      if (coming != patch) {
        // (the first patch, all of its items skipped: a copy that nothing waited for)
        if (coming >= 0) ok = mbar_wait_bounded(&bar[0], nload++ & 1u);
        if (__syncthreads_or(!ok)) {
          if (threadIdx.x == 0) *(volatile int *)P.F.err = kErrTmaTimeout;
          return;
        }
        if (threadIdx.x == 0) issue_copy(patch, tab);
      }
      ok = mbar_wait_bounded(&bar[0], nload++ & 1u);
      coming = -1;
      if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) *(volatile int *)P.F.err = kErrTmaTimeout;
        return;
      }
      cur = patch;
    }
    const int32_t *hdr = reinterpret_cast<const int32_t *>(smem_raw + (tab ? S.tab : L.hdr_off));
    const int nn = hdr[0], own = hdr[1];
    const int n_it = nn * CL;  // staging / output items (node i, pair cl): it = i * CL + cl
    const int cc = c0 + 2 * cl;  // this thread's cases: cc, cc + 1
    T beta[2];
    bool case_done[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      beta[j] = s_beta[cc + j];
      case_done[j] = s_done[cc + j] != 0;
    }
    // 1. stage the chunk's node values: C cases of a node are one contiguous load
    for (int it = threadIdx.x; it < n_it; it += NT) {
      const int i = it / CL;
      const int64_t idx = (int64_t)node(i) * K + cc;
      NodeV<T, VW> v[2], w[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        v[j] = ldv<T, VW>(z, idx + j);
        if (beta[j] != T(0)) w[j] = ldv<T, VW>(pold, idx + j);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (beta[j] != T(0)) {
#pragma unroll
          for (int d = 0; d < DIM; ++d) v[j].v[d] += beta[j] * w[j].v[d];
        }
        // a stopped case keeps its last direction (a continued refinement
        // step starts from it); its lanes still compute, unused
        if (i >= own && !case_done[j]) stv<T, VW>(pnew, idx + j, v[j]);
      }
      const unsigned bb = table(L.bits_off)[i];
      float2 m[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        m[d] = (bb >> d & 1u) ? make_float2(0.f, 0.f) : make_float2(v[0].v[d], v[1].v[d]);
      sp.store(it, m);
    }
    __syncthreads();
    // 2. half-fans: forces relative to P (missing tets have zero gradients),
    //    halves combined by shuffle, written to the force list
    Comp32 energy[2];
#pragma unroll 1
    for (int rd = 0; rd < ROUNDS; ++rd) {
      const int hf = (rd * NW + wid) * HPW + hs;
      int slot[6];
      const int nk = load_half_slots(B + L.slot_off, hf, slot);
      auto force_out = [&](int k, const float2 (&v)[DIM]) {
        if (k < nk && half_writes(h, k)) fs.store(half_fpos(B + L.fpos_off, hf, k) * CL + cl, v);
      };
      auto xor2 = [](float2 v) {
        return make_float2(__shfl_xor_sync(0xffffffffu, v.x, CL), __shfl_xor_sync(0xffffffffu, v.y, CL));
      };
      // The ring vertices go by one after another (a: R_jj, b: R_jj+1), each force
      // written as soon as its two tets are done: 54 registers of node values
      // and forces instead of 72.
      float2 p0[DIM] = {}, dq[DIM] = {}, a[DIM] = {}, fq[DIM] = {}, fa[DIM] = {}, sum[DIM] = {}, r3[DIM];
      if (nk) {
        sp.load(slot[0] * CL + cl, p0);
        sp.load(slot[1] * CL + cl, dq);
        sp.load(slot[2] * CL + cl, a);
      }
      float2 e = make_float2(0.f, 0.f);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        dq[d] = sub2(dq[d], p0[d]);
        a[d] = sub2(a[d], p0[d]);
      }
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) {
        float2 b[DIM] = {}, fb[DIM] = {};
        if (3 + jj < nk) sp.load(slot[3 + jj] * CL + cl, b);
#pragma unroll
        for (int d = 0; d < DIM; ++d) b[d] = sub2(b[d], p0[d]);
        T G[9];
        load_tet_G(B + L.g_off, hf, jj, G);
        tet_forces_acc2(dq, a, b, G, lam, mu, fq, fa, fb);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          sum[d] = __fadd2_rn(sum[d], fa[d]);
          e = __ffma2_rn(a[d], fa[d], e);
          if (jj == 0) r3[d] = xor2(fa[d]);  // half 1's force on R_3, its first ring vertex
        }
        force_out(2 + jj, fa);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          a[d] = b[d];
          fa[d] = fb[d];
        }
      }
      // the forces sum to zero, and sum_k u_k.f_k = sum_k>0 du_k.f_k
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        sum[d] = __fadd2_rn(__fadd2_rn(sum[d], fa[d]), fq[d]);
        e = __ffma2_rn(dq[d], fq[d], __ffma2_rn(a[d], fa[d], e));
        sum[d] = make_float2(-sum[d].x, -sum[d].y);
      }
      energy[0].add(e.x);
      energy[1].add(e.y);
      // half 1's P, Q and R_3 forces go to half 0
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const float2 p = xor2(sum[d]), q1 = xor2(fq[d]);
        if (h == 0) {
          sum[d] = __fadd2_rn(sum[d], p);
          fq[d] = __fadd2_rn(fq[d], q1);
          fa[d] = __fadd2_rn(fa[d], r3[d]);
        }
      }
      force_out(0, sum);
      force_out(1, fq);
      force_out(5, fa);
    }
    const bool change = next < q1 && next / NC != patch;
    if (change) fence_proxy_async();  // reads of the block precede the copy that overwrites it
    __syncthreads();
    if (change) {  // slots, force positions and gradients are done with; the node tables have a second copy
      coming = next / NC;
      if (threadIdx.x == 0) issue_copy(coming, tab ^ 1);
    }
    // 3. node sums over contiguous force runs, constrained DOFs: (I - P) diag(A) p on owned nodes
    for (int it = threadIdx.x; it < n_it; it += NT) {
      const int i = it / CL;
      const unsigned bb = table(L.bits_off)[i];
      float2 acc[DIM] = {};
      const uint16_t *fstart = reinterpret_cast<const uint16_t *>(table(L.fstart_off));
      const int k1 = fstart[i + 1];
#pragma unroll 4
      for (int k = fstart[i]; k < k1; ++k) {
        float2 f[DIM];
        fs.load(k * CL + cl, f);
#pragma unroll
        for (int d = 0; d < DIM; ++d) acc[d] = __fadd2_rn(acc[d], f[d]);
      }
      const int g = node(i);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        NodeV<T, VW> out;
        bool any = false;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          out.v[d] = (bb >> d & 1u) ? T(0) : j ? acc[d].y : acc[d].x;
          any |= out.v[d] != T(0);
        }
        out.v[3] = 0;
        const int64_t idx = (int64_t)g * K + cc + j;
        if ((bb & kBcBits) && i >= own) {
          const NodeV<T, VW> v = ldv<T, VW>(pnew, idx);  // this thread wrote pnew[idx] while staging
          const NodeV<T, VW> dg = ldv<T, VW>(P.diagA, g);
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            if (bb >> d & 1u) {
              const T t = dg.v[d] * v.v[d];
              out.v[d] = t;
              any |= t != T(0);
              energy[j].add(t * v.v[d]);
            }
        }
        if (any) atomic_addv<T, VW>(y, idx, out, DIM);
      }
    }
    // per-case energy of the item: lanes of one case, then warps in order
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int o = CL; o < 32; o <<= 1) {
        const float h2 = __shfl_xor_sync(0xffffffffu, energy[j].hi, o);
        const float l2 = __shfl_xor_sync(0xffffffffu, energy[j].lo, o);
        energy[j].merge(h2, l2);
      }
      if (lane < CL) s_red[wid * C + 2 * lane + j] = make_float2(energy[j].hi, energy[j].lo);
    }
    __syncthreads();  // sp, fs and s_red of this item are complete
    // (a tree of eight lanes per case, in FP64; two warps do it while the others
    // go on. FP64 conversions and sums in every warp before the barrier took
    // a tenth of an item.)
    if (threadIdx.x < 8 * C) {
      const float2 e0 = s_red[(threadIdx.x & 7) * C + (threadIdx.x >> 3)];
      double t = (double)e0.x + (double)e0.y;
      if (NW > 8) {
        const float2 e1 = s_red[((threadIdx.x & 7) + 8) * C + (threadIdx.x >> 3)];
        t += (double)e1.x + (double)e1.y;
      }
      const unsigned mask = C < 4 ? (1u << (8 * (C & 3))) - 1u : 0xffffffffu;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(mask, t, o);
      if ((threadIdx.x & 7) == 0) s_en[c0 + (threadIdx.x >> 3)] += t;
    }
  }
  if (threadIdx.x == 0 && coming >= 0) mbar_wait_bounded(&bar[0], nload & 1u);
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
  griddep_wait();
  griddep_launch_dependents();  // the next matvec may start its first block copies
  // U items per thread per round, all loads issued before any is used; the
  // stride is a multiple of K, so every item of a thread is the same case. The
  // first round's loads are issued before the scalars are formed (an FP64
  // division in one warp takes longer than they do).
  constexpr int U = 4;
  const int64_t n_items = P.n_nodes * K;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  NodeV<T, VW> di[U], rv[U], xx[U], pp[U], uu[U];
  auto load = [&]() {
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
  };
  load();
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
    const int fz = !init && case_stopped(m.done[q]);
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
  for (bool loaded = true; i0 < n_items; i0 += stride * U, loaded = false) {
    NodeV<T, VW> zero;
#pragma unroll
    for (int d = 0; d < VW; ++d) zero.v[d] = 0;
    if (frozen) {
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (i0 + k * stride < n_items) stv<T, VW>(u, i0 + k * stride, zero);
      continue;
    }
    if (!loaded) load();
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

// After the init kernel: the scalars of every case (one block). ref: per case
// ||f||^2 and r.z that the stopping test refers to instead of this run's own
// (0: its own; null: none), the start of a refinement step that goes on, and the
// iterations that this step has taken.
static __global__ void __launch_bounds__(kMaxCases)
    k_multi_start(MultiScalars *sc, MultiCtl *ctl, int K, const double *ref) {
  const int c = threadIdx.x;
  bool stop = true;
  if (c < K) {
    MultiScalars &m = sc[c];
    const double g = m.sum_b[0][0], rr = m.sum_b[0][1], ff = m.sum_a[0];
    const bool resumed = ref && ref[3 * c] > 0;
    const double lim = ctl->tol * sqrt(resumed ? ref[3 * c] : ff);
    m.gamma0 = m.gamma = m.gamma_prev = g;
    m.rr = rr;
    m.ff = ff;
    m.gamma_stop = ctl->tol * (resumed ? ref[3 * c + 1] : g);
    m.cap = ctl->maxit - (resumed ? (int)ref[3 * c + 2] : 0);
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
