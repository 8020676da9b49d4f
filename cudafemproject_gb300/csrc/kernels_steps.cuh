// FP64 time stepping on the assembled node rows (kernels_rows.cuh): explicit
// GN22 steps and the reverse sweep of their adjoint, each a cooperative kernel
// that runs a range of steps with one grid barrier per step, and the modulus
// gradient of a range of steps. The reference's re-sorted lumped masses
// (kernels_aux.cuh) are advanced inside the same kernel, one step ahead.
//
// Two lanes own a row and split its components (as in k_rows_pcg). RESIDENT:
// every warp has at most one slice and the rows' state stays in registers from
// step to step; otherwise it is loaded and stored in every step.
#pragma once

#include "kernels_rows.cuh"

namespace cfem {

constexpr int kStepThreads = 512;
constexpr int kStepWarps = kStepThreads / 32;

// The reference assembles the element masses (or preconditioner diagonals) by
// sorting them by DOF key in place, so every assembly permutes the source of
// the next one: src' = src[perm], and the value of DOF k is the sum of src'
// over its segment, in order. One warp handles 32 DOFs at a time: it gathers
// their slots in contiguous runs (coalesced reads of perm, coalesced writes of
// src'), stages them in shared memory, and each lane adds up its own segment.
constexpr int kResortTile = 768;  // slots staged per warp (24 per DOF of a hex-derived mesh)
struct Resort {
  int64_t n_dof;
  int dim, vw;
  const int64_t *seg;      // [n_dof + 1]
  const int32_t *perm;     // [slots]
  const int32_t *old2new;  // caller node -> node
};

// DOFs [k0, k1) (k1 - k0 <= 32); out: node vector of the sums, or of their
// inverses (0 where the sum is 0). stage: kResortTile doubles of the warp.
template <typename T>
__device__ __forceinline__ void resort_warp(const Resort &R, int64_t k0, int64_t k1, const double *src, double *dst,
                                            T *out, bool invert, double *stage) {
  const int lane = threadIdx.x & 31;
  const int64_t k = k0 + lane;
  const bool mine = k < k1;
  const int64_t j0 = R.seg[k0], j1 = R.seg[k1];
  const int64_t a = mine ? R.seg[k] : j1, b = mine ? R.seg[k + 1] : j1;
  double acc = 0;
  for (int64_t t0 = j0; t0 < j1; t0 += kResortTile) {
    const int64_t t1 = min(t0 + kResortTile, j1);
    int64_t j = t0 + lane;
    for (; j + 96 < t1; j += 128) {  // four gathers in flight
      int32_t p[4];
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) p[q] = __ldcs(R.perm + j + 32 * q);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = src[p[q]];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        dst[j + 32 * q] = v[q];
        stage[j + 32 * q - t0] = v[q];
      }
    }
    for (; j < t1; j += 32) {
      const double v = src[R.perm[j]];
      dst[j] = v;
      stage[j - t0] = v;
    }
    __syncwarp();
    for (int64_t q = max(a, t0); q < min(b, t1); ++q) acc += stage[q - t0];
    __syncwarp();
  }
  if (mine) {
    const int64_t node = k / R.dim, d = k - node * R.dim;
    const double v = invert ? (acc != 0 ? 1.0 / acc : 0.0) : acc;
    out[(int64_t)R.old2new[node] * R.vw + d] = (T)v;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_resort(Resort R, const double *src, double *dst, T *out, int invert) {
  __shared__ double stage[kThreads / 32][kResortTile];
  const int64_t k0 = (blockIdx.x * (int64_t)(kThreads / 32) + (threadIdx.x >> 5)) * 32;
  if (k0 < R.n_dof) resort_warp<T>(R, k0, min(k0 + 32, R.n_dof), src, dst, out, invert != 0, stage[threadIdx.x >> 5]);
}

// ------------------------------------------------------------------ explicit steps
// d_n = d_{n-1} + dt v + c2 a; a_n = (F(t_n) - K' d_n) / M;
// v += c_old a_{n-1} + c_new a_n, for n = first .. last.
struct RowsSteps {
  RowOp A;
  int first, last;
  double *v, *a;              // state after step first - 1 in, after step last out
  double *d;                  // d_n at d + ((n - n0) & mask) * stride; d_{first-1} in, d_last out
  int n0, mask;
  int64_t stride;
  const double *FA, *FB, *coef;  // F(t_n) = coef[2n] FA + coef[2n+1] FB
  const double *minv;         // inverse lumped masses; re-sorted: two node vectors, step n uses n & 1
  double dt, c2, c_old, c_new;
  int resort;
  Resort R;
  double *src[2];             // re-sorted: the source before step n in src[(n - first) & 1]
  double *minv2[2];
  int n_recv, dim;            // d_n of the receivers into trace[n - 1]
  const int32_t *recv;
  double *trace;
  GridSync sync;
  int *stalled;
};

template <int DIM, bool RESIDENT, bool WIDE = false>
__global__ void __launch_bounds__(kStepThreads, 1) k_rows_steps(RowsSteps P) {
  constexpr int VW = DIM == 3 ? 4 : 2;
  constexpr int OWN = DIM == 3 ? 2 : 1;
  extern __shared__ double stage_raw[];  // re-sorting: kResortTile per warp
  __shared__ GridShared<128> sh;
  if (P.sync.absent_plus1 == (int)blockIdx.x + 1) return;  // (self-test of the waits for it)
  const RowOp &A = P.A;
  const int wid = threadIdx.x >> 5, half = (threadIdx.x >> 4) & 1;
  const int64_t s0 = A.n_slices * blockIdx.x / gridDim.x, s1 = A.n_slices * (blockIdx.x + 1) / gridDim.x;
  const int c0 = half * OWN, n_own = DIM - c0 < OWN ? DIM - c0 : OWN;
  unsigned epoch = 0;
  auto dn = [&](int n) { return P.d + (int64_t)((n - P.n0) & P.mask) * P.stride; };
  auto resort_all = [&](int n) {  // masses of step n
    double *stage = stage_raw + (size_t)wid * kResortTile;
    const int64_t groups = (P.R.n_dof + 31) / 32;
    const int64_t g0 = groups * blockIdx.x / gridDim.x, g1 = groups * (blockIdx.x + 1) / gridDim.x;
    const int64_t k1 = min(P.R.n_dof, g1 * 32);
    for (int64_t k = (g0 + wid) * 32; k < k1; k += 32 * kStepWarps)
      resort_warp<double>(P.R, k, min(k + 32, k1), P.src[(n - P.first) & 1], P.src[(n - P.first + 1) & 1],
                          P.minv2[n & 1], true, stage);
  };
  // the lane's components of its row (RESIDENT: kept; else of the slice at hand)
  int row = -1;
  double d[DIM], v[OWN], a[OWN], fa[OWN], fb[OWN], mi[OWN];
  bool loaded = false;  // some row of the slice has a load
  auto load_state = [&](int64_t s, const double *from) {
    row = rows_own<DIM>(A, s, from, d);
    loaded = false;
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      v[k] = a[k] = fa[k] = fb[k] = mi[k] = 0;
      if (row >= 0 && k < n_own) {
        const int64_t i = (int64_t)row * VW + c0 + k;
        v[k] = P.v[i];
        a[k] = P.a[i];
        fa[k] = P.FA[i];
        fb[k] = P.FB[i];
        if (!P.resort) mi[k] = P.minv[i];
        loaded |= fa[k] != 0 || fb[k] != 0;
      }
    }
    loaded = __any_sync(0xffffffffu, loaded);
  };
  auto store_state = [&]() {
#pragma unroll
    for (int k = 0; k < OWN; ++k)
      if (row >= 0 && k < n_own) {
        const int64_t i = (int64_t)row * VW + c0 + k;
        P.v[i] = v[k];
        P.a[i] = a[k];
      }
  };
  auto predict = [&](double *to) {  // d_{n+1} from the state after step n
    double o[OWN];
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const double mine = half ? (OWN + k < DIM ? d[OWN + k < DIM ? OWN + k : 0] : 0.0) : d[k];
      o[k] = fma(P.c2, a[k], fma(P.dt, v[k], mine));
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const double other = __shfl_xor_sync(0xffffffffu, o[k], 16);
      d[k] = half ? other : o[k];
      if (OWN + k < DIM) d[OWN + k < DIM ? OWN + k : 0] = half ? o[k] : other;
    }
    if (row >= 0 && !half) {
      NodeV<double, VW> w;
#pragma unroll
      for (int q = 0; q < VW; ++q) w.v[q] = q < DIM ? d[q < DIM ? q : 0] : 0.0;
      stv<double, VW>(to, row, w);
    }
  };
  const bool mine = RESIDENT && s0 + wid < s1;
  // d_first, and the masses of the first step
  if constexpr (RESIDENT) {
    if (mine) {
      load_state(s0 + wid, dn(P.first - 1));
      predict(dn(P.first));
    }
  } else {
    for (int64_t s = s0 + wid; s < s1; s += kStepWarps) {
      load_state(s, dn(P.first - 1));
      predict(dn(P.first));
    }
  }
  if (P.resort) resort_all(P.first);
  for (int n = P.first; n <= P.last; ++n) {
    if (!grid_barrier(P.sync, ++epoch, sh)) {
      if (threadIdx.x == 0) atomicExch(P.stalled, 1);
      return;
    }
    const double *cur = dn(n);
    const double ca = P.coef[2 * n], cb = P.coef[2 * n + 1];
    const bool finite = isfinite(ca) && isfinite(cb);
    const double *m = P.resort ? P.minv2[n & 1] : P.minv;
    if (blockIdx.x == gridDim.x - 1)
      for (int i = threadIdx.x; i < P.n_recv * P.dim; i += kStepThreads) {
        const int r = i / P.dim, k = i % P.dim;
        P.trace[((int64_t)(n - 1) * P.n_recv + r) * P.dim + k] = cur[(int64_t)P.recv[r] * VW + k];
      }
    auto step = [&](int64_t s) {
      double y[DIM];
      rows_product<DIM, WIDE>(A, s, row, cur, d, y);
#pragma unroll
      for (int k = 0; k < OWN; ++k) {
        const double yk = half ? (OWN + k < DIM ? y[OWN + k < DIM ? OWN + k : 0] : 0.0) : y[k];
        if (P.resort && row >= 0 && k < n_own) mi[k] = m[(int64_t)row * VW + c0 + k];
        const double f = loaded || !finite ? fma(ca, fa[k], cb * fb[k]) - yk : -yk;
        const double an = f * mi[k];
        v[k] = fma(P.c_new, an, fma(P.c_old, a[k], v[k]));
        a[k] = an;
      }
      if (n < P.last) predict(dn(n + 1));
    };
    // (half of the warps of every SM quarter re-sort first, so that one half's
    // gathers overlap the other half's products)
    const bool resort = P.resort && n < P.last, early = (wid >> 2) & 1;
    if (resort && early) resort_all(n + 1);
    if constexpr (RESIDENT) {
      if (mine) step(s0 + wid);
    } else {
      for (int64_t s = s0 + wid; s < s1; s += kStepWarps) {
        load_state(s, cur);
        step(s);
        store_state();
      }
    }
    if (resort && !early) resort_all(n + 1);
  }
  if constexpr (RESIDENT) {
    if (mine) store_state();
  }
}

// ------------------------------------------------------------------ reverse sweep
// Adjoint of the steps last .. first: db += d_n - obs_n at the receivers;
// w_n = (ab + h_new vb) / M; ab = h_old vb; db -= K' w_n; vb += dt db;
// ab += c2 db.
struct RowsReverse {
  RowOp A;
  int first, last;
  double *db, *vb, *ab;
  const double *d;            // d_n at d + (n - n0) * stride
  double *w;                  // w_n at w + (n - n0) * stride
  int n0;
  int64_t stride;
  const double *minv;
  double dt, c2, h_old, h_new;
  const int32_t *rec_head, *rec_next;  // receivers at a node: rec_head[node] (-1: none), rec_next[r]
  int n_rec;
  const double *obs;          // [n - 1][n_rec][DIM]
  GridSync sync;
  int *stalled;
};

template <int DIM, bool RESIDENT, bool WIDE = false>
__global__ void __launch_bounds__(kStepThreads, 1) k_rows_reverse(RowsReverse P) {
  constexpr int VW = DIM == 3 ? 4 : 2;
  constexpr int OWN = DIM == 3 ? 2 : 1;
  __shared__ GridShared<128> sh;
  if (P.sync.absent_plus1 == (int)blockIdx.x + 1) return;  // (self-test of the waits for it)
  const RowOp &A = P.A;
  const int wid = threadIdx.x >> 5, half = (threadIdx.x >> 4) & 1;
  const int64_t s0 = A.n_slices * blockIdx.x / gridDim.x, s1 = A.n_slices * (blockIdx.x + 1) / gridDim.x;
  const int c0 = half * OWN, n_own = DIM - c0 < OWN ? DIM - c0 : OWN;
  unsigned epoch = 0;
  int row = -1, head = -1;
  double w[DIM], db[OWN], vb[OWN], ab[OWN], mi[OWN];
  auto load_state = [&](int64_t s) {
    row = A.row[s * kSliceRows + (threadIdx.x & 15)];
    head = row >= 0 ? P.rec_head[row] : -1;
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      db[k] = vb[k] = ab[k] = mi[k] = 0;
      if (row >= 0 && k < n_own) {
        const int64_t i = (int64_t)row * VW + c0 + k;
        db[k] = P.db[i];
        vb[k] = P.vb[i];
        ab[k] = P.ab[i];
        mi[k] = P.minv[i];
      }
    }
  };
  auto store_state = [&]() {
#pragma unroll
    for (int k = 0; k < OWN; ++k)
      if (row >= 0 && k < n_own) {
        const int64_t i = (int64_t)row * VW + c0 + k;
        P.db[i] = db[k];
        P.vb[i] = vb[k];
        P.ab[i] = ab[k];
      }
  };
  auto before = [&](int n) {  // receivers, w_n, ab
    for (int r = head; r >= 0; r = P.rec_next[r])
#pragma unroll
      for (int k = 0; k < OWN; ++k)
        if (k < n_own)
          db[k] += P.d[(int64_t)(n - P.n0) * P.stride + (int64_t)row * VW + c0 + k] -
                   P.obs[((int64_t)(n - 1) * P.n_rec + r) * DIM + c0 + k];
    double o[OWN];
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      o[k] = fma(P.h_new, vb[k], ab[k]) * mi[k];
      ab[k] = P.h_old * vb[k];
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const double other = __shfl_xor_sync(0xffffffffu, o[k], 16);
      w[k] = half ? other : o[k];
      if (OWN + k < DIM) w[OWN + k < DIM ? OWN + k : 0] = half ? o[k] : other;
    }
    if (row >= 0 && !half) {
      NodeV<double, VW> t;
#pragma unroll
      for (int q = 0; q < VW; ++q) t.v[q] = q < DIM ? w[q < DIM ? q : 0] : 0.0;
      stv<double, VW>(P.w + (int64_t)(n - P.n0) * P.stride, row, t);
    }
  };
  auto after = [&](int64_t s, int n) {
    double y[DIM];
    rows_product<DIM, WIDE>(A, s, row, P.w + (int64_t)(n - P.n0) * P.stride, w, y);
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const double yk = half ? (OWN + k < DIM ? y[OWN + k < DIM ? OWN + k : 0] : 0.0) : y[k];
      db[k] -= yk;
      vb[k] = fma(P.dt, db[k], vb[k]);
      ab[k] = fma(P.c2, db[k], ab[k]);
    }
  };
  const bool mine = RESIDENT && s0 + wid < s1;
  if constexpr (RESIDENT) {
    if (mine) load_state(s0 + wid);
  }
  for (int n = P.last; n >= P.first; --n) {
    if constexpr (RESIDENT) {
      if (mine) before(n);
    } else {
      for (int64_t s = s0 + wid; s < s1; s += kStepWarps) {
        load_state(s);
        before(n);
        store_state();
      }
    }
    if (!grid_barrier(P.sync, ++epoch, sh)) {
      if (threadIdx.x == 0) atomicExch(P.stalled, 1);
      return;
    }
    if constexpr (RESIDENT) {
      if (mine) after(s0 + wid, n);
    } else {
      for (int64_t s = s0 + wid; s < s1; s += kStepWarps) {
        load_state(s);
        rows_own<DIM>(A, s, P.w + (int64_t)(n - P.n0) * P.stride, w);
        after(s, n);
        store_state();
      }
    }
  }
  if constexpr (RESIDENT) {
    if (mine) store_state();
  }
}

// ------------------------------------------------------------------ modulus gradient
// g_e -= (1 / E_e) sum_n w_n^T (K'_e) u_n over the unconstrained DOFs plus the
// diagonal terms of the constrained ones, for `count` pairs of node vectors
// (u + k * stride, w + k * stride). One thread per element and every SPLIT-th
// pair (the four warps of a block share 32 elements when there are many pairs,
// which evens out the FP64 work over the SM quarters of a small mesh), its
// gradients read once for all its pairs; with H the displacement gradient scaled by
// sqrt(V E_e / E), w^T K_e u = lam tr(H_u) tr(H_w) + 2 mu sym(H_u) : sym(H_w).
template <int DIM, int SPLIT>
__global__ void __launch_bounds__(128) k_grad_pairs(int64_t ne, const double *G64, int64_t gstride, const int32_t *conn,
                                                    const uint8_t *bits, double lam, double mu, const double *u,
                                                    const double *w, int64_t stride, int count, const double *young,
                                                    const int32_t *elem_new2old, double *g_out, int accumulate) {
  constexpr int NV = DIM + 1, VW = DIM == 3 ? 4 : 2;
  __shared__ double part[128];
  const int part_of = SPLIT == 1 ? 0 : threadIdx.x >> 5;
  const int64_t ei = SPLIT == 1 ? blockIdx.x * (int64_t)128 + threadIdx.x : blockIdx.x * (int64_t)32 + (threadIdx.x & 31);
  const int64_t e = ei < ne ? ei : ne - 1;
  double G[DIM * DIM];
#pragma unroll
  for (int k = 0; k < DIM * DIM; ++k) G[k] = G64[(size_t)k * gstride + e];
  int node[NV];
  unsigned b[NV], any = 0;
#pragma unroll
  for (int a = 0; a < NV; ++a) {
    node[a] = conn[e * NV + a];
    b[a] = bits[node[a]];
    any |= b[a];
  }
  double acc = 0;
  for (int k = part_of; k < count; k += SPLIT) {
    const double *uk = u + k * stride, *wk = w + k * stride;
    double H[DIM][DIM], Q[DIM][DIM];
    auto gradient = [&](const double *x, double (&h)[DIM][DIM]) {
      double x0[DIM];
#pragma unroll
      for (int i = 0; i < DIM; ++i)
#pragma unroll
        for (int j = 0; j < DIM; ++j) h[i][j] = 0;
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        NodeV<double, VW> t = ldv<double, VW>(x, node[a]);
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
          const double xi = (b[a] >> i) & 1u ? 0.0 : t.v[i];
          if (a == 0) {
            x0[i] = xi;
          } else {
            const double dx = xi - x0[i];
#pragma unroll
            for (int j = 0; j < DIM; ++j) h[i][j] = fma(dx, G[(a > 0 ? a - 1 : 0) * DIM + j], h[i][j]);
          }
        }
      }
    };
    gradient(uk, H);
    gradient(wk, Q);
    double tu = 0, tw = 0, diag = 0, shear = 0;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      tu += H[i][i];
      tw += Q[i][i];
      diag = fma(H[i][i], Q[i][i], diag);
#pragma unroll
      for (int j = i + 1; j < DIM; ++j) shear = fma(H[i][j] + H[j][i], Q[i][j] + Q[j][i], shear);
    }
    acc += fma(lam * tu, tw, mu * fma(2.0, diag, shear));
    if (any) {
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        if (!b[a]) continue;
        double sq[DIM], tot = 0;
#pragma unroll
        for (int i = 0; i < DIM; ++i) {
          double gi = 0;
          if (a == 0) {
#pragma unroll
            for (int q = 0; q < DIM; ++q) gi -= G[q * DIM + i];
          } else {
            gi = G[(a > 0 ? a - 1 : 0) * DIM + i];
          }
          sq[i] = gi * gi;
          tot += sq[i];
        }
#pragma unroll
        for (int i = 0; i < DIM; ++i)
          if ((b[a] >> i) & 1u) {
            const double kd = (lam + 2 * mu) * sq[i] + mu * (tot - sq[i]);
            acc += wk[(int64_t)node[a] * VW + i] * kd * uk[(int64_t)node[a] * VW + i];
          }
      }
    }
  }
  if constexpr (SPLIT > 1) {
    part[threadIdx.x] = acc;
    __syncthreads();
    if (part_of) return;
#pragma unroll
    for (int q = 1; q < SPLIT; ++q) acc += part[q * 32 + threadIdx.x];
  }
  if (ei >= ne) return;
  const int64_t eo = elem_new2old[e];
  const double v = -acc / young[eo];
  g_out[eo] = accumulate ? g_out[eo] + v : v;
}

}  // namespace cfem
