// FP64 operator as assembled node rows.
//
// GB300's FP64 pipe is narrow (about 2 lanes per SM and cycle), and the FP64
// element kernels were bound by it: 97 FP64 operations per tetrahedron, 580 per
// node of a hex-derived mesh. Summed per node pair, the same operator costs 12
// per neighbour, 168 per node (14 neighbours): y_i = sum_j K_ij (x_j - x_i).
// The difference form needs no diagonal block (the rows of a stiffness sum to
// zero) and rounds relative to the displacement differences, like the element
// form; K_ij x_j with the diagonal block would be 135 operations, but its
// rounding is relative to the displacements themselves, which raises the floor
// of the true residual by the ratio of the two (about the number of elements
// along the body).
//
// Constraints: K' = P K P + (I - P) diag(K). Stored blocks are P_i K_ij P_j;
// what the difference form misses next to constrained DOFs, and the diagonal
// of the constrained DOFs themselves, is a small block D_i per node, read only
// by the row slices that need it (a flag per slice).
//
// Layout: rows are sorted by their neighbour count within windows of kRowWindow
// nodes and cut into slices of 16 rows, one warp per slice, two lanes per row:
// lane = 16 * half + r holds neighbours half, half + 2, ... of row r. Step k of
// a slice is 32 column ids and, per block component, 32 doubles: every load of
// the operator is one contiguous 256-byte line per warp. Unused entries repeat
// the row itself (difference zero). A node of more than kWideDegree neighbours has
// a slice of its own (kWideSlice), in which lane l holds neighbours l, l + 32, ..:
// two lanes took 0.57 ms for a product with 1000 neighbours, 5.4 with 10,000
// (element form 0.09 and 0.10), a warp 0.06 and 0.30.
#pragma once

#include "grid_sync.cuh"
#include "kernels.cuh"

namespace cfem {

constexpr int kRowWindow = 512;  // nodes among which rows are sorted by neighbour count
constexpr int kSliceRows = 16;
constexpr int kWideDegree = 64;  // (16 rows of 64 neighbours: 32 steps; meshes of tetrahedra have 15 to 35)
constexpr unsigned kHasD = 1, kWideSlice = 2;  // RowOp::flag

struct RowOp {
  int64_t n_slices;
  const int64_t *off;   // [n_slices + 1] first step of each slice
  const int32_t *row;   // [n_slices][16] node, or -1
  const int32_t *col;   // [steps][32]
  const double *val;    // [steps][DIM * DIM][32]
  const uint8_t *flag;  // [n_slices] kHasD: rows with a D block; kWideSlice: one row
  const double *D;      // [n_nodes][DIM * DIM]
  const uint8_t *bits;  // [n_nodes] constrained DOFs
};

// Where a row product reads x: a node vector, or the caller's [n_nodes][DIM].
template <int DIM>
struct NodeX {
  static constexpr int VW = DIM == 3 ? 4 : 2;
  const double *x;
  __device__ __forceinline__ NodeV<double, VW> operator()(int32_t j) const { return ldv<double, VW>(x, j); }
};
template <int DIM>
struct CallerX {
  static constexpr int VW = DIM == 3 ? 4 : 2;
  const double *x;
  const int32_t *new2old;
  __device__ __forceinline__ NodeV<double, VW> operator()(int32_t j) const {
    const double *p = x + (int64_t)new2old[j] * DIM;
    NodeV<double, VW> v;
#pragma unroll
    for (int d = 0; d < VW; ++d) v.v[d] = d < DIM ? p[d < DIM ? d : 0] : 0.0;
    return v;
  }
};

template <int DIM, bool MASKED, typename X>
__device__ __forceinline__ void rows_sum(const RowOp &A, int64_t k0, int n, const X &x, const double (&xi)[DIM],
                                         double (&y)[DIM]) {
  constexpr int VW = DIM == 3 ? 4 : 2, NC = DIM * DIM;
  const int32_t *col = A.col + k0 * 32 + (threadIdx.x & 31);
  const double *val = A.val + k0 * (32 * NC) + (threadIdx.x & 31);
#pragma unroll 2
  for (int k = 0; k < n; ++k) {
    double K[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) K[c] = __ldcs(val + (k * NC + c) * 32);
    const int32_t j = col[k * 32];
    NodeV<double, VW> v = x(j);
    if (MASKED) {  // values at constrained DOFs have no influence, whatever they are
      const unsigned b = A.bits[j];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        if ((b >> d) & 1u) v.v[d] = 0;
    }
    double du[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) du[d] = v.v[d] - xi[d];
#pragma unroll
    for (int p = 0; p < DIM; ++p)
#pragma unroll
      for (int q = 0; q < DIM; ++q) y[p] = fma(K[p * DIM + q], du[q], y[p]);
  }
#pragma unroll
  for (int d = 0; d < DIM; ++d) y[d] += __shfl_xor_sync(0xffffffffu, y[d], 16);
}

// y = A x for the rows of slice s, given the rows (-1: padding) and their own
// x; both lanes of a row get the sum. x is read with plain loads: callers may
// have other CTAs' writes made visible by a grid barrier. WIDE: the operator has
// slices of one row (instances of their own: the test for them in every product
// took 4% of the time steps).
template <int DIM, bool WIDE, typename X>
__device__ __forceinline__ void rows_product_of(const RowOp &A, int64_t s, int row, const X &x,
                                                const double (&xi)[DIM], double (&y)[DIM]) {
  constexpr int NC = DIM * DIM;
  const int64_t k0 = A.off[s];
  const int n = (int)(A.off[s + 1] - k0);
#pragma unroll
  for (int d = 0; d < DIM; ++d) y[d] = 0;
  const unsigned flag = A.flag[s];
  if (!flag) {
    rows_sum<DIM, false>(A, k0, n, x, xi, y);
    return;
  }
  double xr[DIM], xm[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) xr[d] = xi[d];
  int i = row < 0 ? 0 : row;
  const bool wide = WIDE && (flag & kWideSlice);
  if (wide) {  // every lane works for the row of lanes 0 and 16
    i = __shfl_sync(0xffffffffu, row, 0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) xr[d] = __shfl_sync(0xffffffffu, xi[d], 0);
  }
  const unsigned b = A.bits[i];
#pragma unroll
  for (int d = 0; d < DIM; ++d) xm[d] = (b >> d) & 1u ? 0.0 : xr[d];
  rows_sum<DIM, true>(A, k0, n, x, xm, y);
  if (wide)
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int d = 0; d < DIM; ++d) y[d] += __shfl_xor_sync(0xffffffffu, y[d], o);
  const double *D = A.D + (int64_t)i * NC;
#pragma unroll
  for (int p = 0; p < DIM; ++p) {
    if ((b >> p) & 1u) {
      y[p] = D[p * DIM + p] * xr[p];
    } else {
#pragma unroll
      for (int q = 0; q < DIM; ++q) y[p] = fma(D[p * DIM + q], xm[q], y[p]);
    }
  }
}

template <int DIM, bool WIDE>
__device__ __forceinline__ void rows_product(const RowOp &A, int64_t s, int row, const double *x,
                                             const double (&xi)[DIM], double (&y)[DIM]) {
  rows_product_of<DIM, WIDE>(A, s, row, NodeX<DIM>{x}, xi, y);
}

// row of this lane in slice s and its own x
template <int DIM>
__device__ __forceinline__ int rows_own(const RowOp &A, int64_t s, const double *x, double (&xi)[DIM]) {
  constexpr int VW = DIM == 3 ? 4 : 2;
  const int row = A.row[s * kSliceRows + (threadIdx.x & 15)];
  const NodeV<double, VW> own = ldv<double, VW>(x, row < 0 ? 0 : row);
#pragma unroll
  for (int d = 0; d < DIM; ++d) xi[d] = own.v[d];
  return row;
}

// ------------------------------------------------------------------ applications
// Four slices per CTA, one for the FP64 pipe of each SM quarter; more would
// leave SMs of a small mesh without any (2601 nodes: 41 CTAs).
constexpr int kRowsThreads = 128;

// y = A x; CALLER: x and y are the caller's [n_nodes][DIM] arrays (not
// overlapping), else node vectors.
template <int DIM, bool CALLER, bool WIDE>
__global__ void __launch_bounds__(kRowsThreads) k_rows_apply(RowOp A, const double *x, double *y, const int32_t *new2old) {
  constexpr int VW = DIM == 3 ? 4 : 2;
  const int64_t s = blockIdx.x * (int64_t)(kRowsThreads / 32) + (threadIdx.x >> 5);
  if (s >= A.n_slices) return;
  double v[DIM], xi[DIM];
  const int row = A.row[s * kSliceRows + (threadIdx.x & 15)];
  auto product = [&](const auto &X) {
    const NodeV<double, VW> own = X(row < 0 ? 0 : row);
#pragma unroll
    for (int d = 0; d < DIM; ++d) xi[d] = own.v[d];
    rows_product_of<DIM, WIDE>(A, s, row, X, xi, v);
  };
  if constexpr (CALLER) product(CallerX<DIM>{x, new2old});
  else product(NodeX<DIM>{x});
  if (row < 0 || (threadIdx.x & 16)) return;
  if constexpr (CALLER) {
    const int64_t o = new2old[row];
#pragma unroll
    for (int d = 0; d < DIM; ++d) y[o * DIM + d] = v[d];
  } else {
    NodeV<double, VW> o;
#pragma unroll
    for (int d = 0; d < VW; ++d) o.v[d] = d < DIM ? v[d < DIM ? d : 0] : 0.0;
    stv<double, VW>(y, row, o);
  }
}

// r = f - A x (x == nullptr: r = f), its FP32 copy, ||r||^2 and ||f||^2 into
// out[0], out[1] (partials: [grid][2], block order).
struct RowsResidual {
  int64_t nn;
  const double *f, *x;
  double *r;
  float *r32;  // or nullptr
  double *out, *partials;
  unsigned int *count;
};
template <int DIM, bool WIDE>
__global__ void __launch_bounds__(kRowsThreads) k_rows_residual(RowOp A, RowsResidual P) {
  constexpr int VW = DIM == 3 ? 4 : 2;
  double acc[2] = {0, 0};
  const int64_t W = (int64_t)gridDim.x * (kRowsThreads / 32);
  for (int64_t s = blockIdx.x * (int64_t)(kRowsThreads / 32) + (threadIdx.x >> 5); s < A.n_slices; s += W) {
    double v[DIM], xi[DIM];
    int row;
    if (P.x) {
      row = rows_own<DIM>(A, s, P.x, xi);
      rows_product<DIM, WIDE>(A, s, row, P.x, xi, v);
    } else {
      row = A.row[s * kSliceRows + (threadIdx.x & 15)];
#pragma unroll
      for (int d = 0; d < DIM; ++d) v[d] = 0;
    }
    if (row < 0 || (threadIdx.x & 16)) continue;
    const NodeV<double, VW> f = ldv<double, VW>(P.f, row);
    NodeV<double, VW> r;
    NodeV<float, VW> r32;
#pragma unroll
    for (int d = 0; d < VW; ++d) {
      r.v[d] = d < DIM ? f.v[d] - v[d < DIM ? d : 0] : 0.0;
      r32.v[d] = (float)r.v[d];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      acc[0] += r.v[d] * r.v[d];
      acc[1] += f.v[d] * f.v[d];
    }
    stv<double, VW>(P.r, row, r);
    if (P.r32) stv<float, VW>(P.r32, row, r32);
  }
  if (grid_sum_last<2>(acc, P.partials, P.count)) {
    P.out[0] = acc[0];
    P.out[1] = acc[1];
  }
}

// FP64 true residuals of K load cases at once: r_c = f_c - A x_c on
// [node][K][4] arrays (3D), ||r_c||^2 and ||f_c||^2 added to norms[2c], [2c + 1]
// (zero at the start). One thread per (row, case), the case fastest: a warp's
// block loads are broadcasts and its gathers contiguous, and the FP64 pipe is
// what bounds it (168 operations per row and case). Cases with skip[c] != 0 are
// left out where a whole warp holds only such. Blocks of 256 threads, K a power
// of two up to 256.
struct RowsCases {
  RowOp A;
  int K;
  const double *f, *x;
  double *r, *norms;
  const int *skip;
};
static __global__ void __launch_bounds__(kThreads) k_rows_cases_residual(RowsCases P) {
  constexpr int DIM = 3;
  const RowOp &A = P.A;
  const int K = P.K, c = threadIdx.x & (K - 1);  // (the grid stride is a multiple of K)
  const bool skip = __all_sync(0xffffffffu, P.skip[c] != 0);
  double rr = 0, ff = 0;
  const int64_t n_items = A.n_slices * kSliceRows * K, stride = (int64_t)gridDim.x * kThreads;
  for (int64_t it = blockIdx.x * (int64_t)kThreads + threadIdx.x; it < n_items && !skip; it += stride) {
    const int64_t slot = it / K, s = slot / kSliceRows;
    const int t = (int)(slot % kSliceRows), row = A.row[slot], i = row < 0 ? 0 : row;
    const int64_t k0 = A.off[s];
    const int n = (int)(A.off[s + 1] - k0);
    const unsigned flag = A.flag[s];
    const bool masked = flag != 0, wide = flag & kWideSlice;
    if (wide && row < 0) continue;
    const unsigned b = masked ? A.bits[i] : 0u;
    NodeV<double, 4> own = ldv<double, 4>(P.x, (int64_t)i * K + c);
    double xi[DIM], y[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      xi[d] = (b >> d) & 1u ? 0.0 : own.v[d];
      y[d] = 0;
    }
    const int32_t *col = A.col + k0 * 32 + t;
    const double *val = A.val + k0 * (32 * DIM * DIM) + t;
    const int n_here = wide ? 16 * n : n;  // (a slice of one row: entry by entry)
    for (int kk = 0; kk < n_here; ++kk)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int k = wide ? kk >> 4 : kk, at = half * 16 + (wide ? kk & 15 : 0);
        const int32_t j = col[k * 32 + at];
        NodeV<double, 4> v = ldv<double, 4>(P.x, (int64_t)j * K + c);
        if (masked) {
          const unsigned bj = A.bits[j];
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            if ((bj >> d) & 1u) v.v[d] = 0;
        }
        double M[DIM * DIM];
#pragma unroll
        for (int q = 0; q < DIM * DIM; ++q) M[q] = val[(k * DIM * DIM + q) * 32 + at];
#pragma unroll
        for (int q = 0; q < DIM; ++q) {
          const double du = v.v[q] - xi[q];
#pragma unroll
          for (int p = 0; p < DIM; ++p) y[p] = fma(M[p * DIM + q], du, y[p]);
        }
      }
    if (masked) {
      const double *Db = A.D + (int64_t)i * DIM * DIM;
#pragma unroll
      for (int p = 0; p < DIM; ++p) {
        if ((b >> p) & 1u) {
          y[p] = Db[p * DIM + p] * own.v[p];
        } else {
#pragma unroll
          for (int q = 0; q < DIM; ++q) y[p] = fma(Db[p * DIM + q], xi[q], y[p]);
        }
      }
    }
    if (row < 0) continue;
    const NodeV<double, 4> f = ldv<double, 4>(P.f, (int64_t)i * K + c);
    NodeV<double, 4> r;
#pragma unroll
    for (int d = 0; d < 4; ++d) r.v[d] = d < DIM ? f.v[d] - y[d < DIM ? d : 0] : 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      rr += r.v[d] * r.v[d];
      ff += f.v[d] * f.v[d];
    }
    stv<double, 4>(P.r, (int64_t)i * K + c, r);
  }
  __shared__ double red[2][kThreads];
  red[0][threadIdx.x] = rr;
  red[1][threadIdx.x] = ff;
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * K; t += kThreads) {
    const int cc = t >> 1, k = t & 1;
    double v = 0;
    for (int q = cc; q < kThreads; q += K) v += red[k][q];
    if (v != 0) atomicAdd(P.norms + t, v);
  }
}

// ------------------------------------------------------------------ Jacobi PCG
// A whole FP64 PCG run in one cooperative kernel: the rows' products and the
// vector updates alternate with grid-wide sums (grid_sync.cuh) instead of
// kernel boundaries, and the run ends in the iteration that meets the stopping
// rule. Per iteration: the sum p.Ap; the sums r.z and r.r; a barrier behind
// which the new direction can be read.
// RESIDENT: every warp has at most one slice, whose rows' x, r, p and M^-1
// stay in registers for the whole run; only p goes through memory, for the
// neighbours. The two lanes of a row share its components (kOwn of them each:
// 0 and 1 in the lower half, 2 in the upper; in 2D one each), because an FP64
// instruction costs the same whatever lanes are active. Otherwise the rows of
// A p and the vectors go through memory.
struct RowsPcg {
  RowOp A;
  const double *f, *dinv;
  double *x, *r, *z, *p, *u;  // RESIDENT: x and p only
  Scalars *sc;                // tol, rule, maxit in; the run's scalars out
  GridSync sync;              // kRowsPcgSets sets of slots
  int warm;                   // start from x
};
// Threads: 512 fill the FP64 pipe and hide the loads; 128, where no CTA has
// more than four slices, shorten every sum by three FP64 additions.
constexpr int kRowsPcgThreads = 512, kRowsPcgSmall = 128;
constexpr int kRowsPcgSets = 5;  // one for the start; of even and of odd iterations, p.Ap and r.z with r.r

template <int DIM, bool RESIDENT, int THREADS, bool WIDE = false>
__global__ void __launch_bounds__(THREADS, 1) k_rows_pcg(RowsPcg P) {
  constexpr int WARPS = THREADS / 32;
  constexpr int VW = DIM == 3 ? 4 : 2;
  constexpr int OWN = DIM == 3 ? 2 : 1;
  __shared__ GridShared<THREADS> sh;
  const GridSync &G = P.sync;
  if (G.absent_plus1 == (int)blockIdx.x + 1) return;  // (self-test of the waits for it)
  const RowOp &A = P.A;
  const int wid = threadIdx.x >> 5, half = (threadIdx.x >> 4) & 1;
  // the CTA's slices, neighbours in node order
  const int64_t s0 = A.n_slices * blockIdx.x / gridDim.x, s1 = A.n_slices * (blockIdx.x + 1) / gridDim.x;
  // not RESIDENT: the nodes of the same slices, so that every vector but p
  // stays with one CTA
  auto each_node = [&](auto &&body) {
    for (int64_t t = s0 * kSliceRows + threadIdx.x; t < s1 * kSliceRows; t += THREADS) {
      const int n = A.row[t];
      if (n >= 0) body(n);
    }
  };
  unsigned epoch = 0;
  auto stalled = [&]() {
    if (threadIdx.x == 0) atomicExch(&P.sc->stalled, 1);
  };
  const double tol = P.sc->tol;
  const int rule = P.sc->rule, maxit = P.sc->maxit;
  // RESIDENT state: the whole p of the lane's row, the components c0 + k of the others
  const int64_t s = s0 + wid;
  const bool mine = RESIDENT && s < s1;
  const int c0 = half * OWN;  // (3D: component 3 of the upper half is a zero)
  int row = -1;
  double x[OWN], r[OWN], m[OWN], p[DIM], y[DIM], yo[OWN];
  auto own_of = [&](const double (&v)[DIM], double (&o)[OWN]) {
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      o[k] = half ? (OWN + k < DIM ? v[OWN + k < DIM ? OWN + k : 0] : 0.0) : v[k];
    }
  };
  // the whole direction of the row from both lanes' components
  auto share_p = [&](const double (&o)[OWN]) {
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const double other = __shfl_xor_sync(0xffffffffu, o[k], 16);
      p[k] = half ? other : o[k];
      if (OWN + k < DIM) p[OWN + k < DIM ? OWN + k : 0] = half ? o[k] : other;
    }
  };
  auto store_p = [&]() {
    if (row < 0 || half) return;
    NodeV<double, VW> pv;
#pragma unroll
    for (int d = 0; d < VW; ++d) pv.v[d] = d < DIM ? p[d < DIM ? d : 0] : 0.0;
    stv<double, VW>(P.p, row, pv);
  };
  double sums[3] = {0, 0, 0};  // r.z, r.r, f.f
  if constexpr (RESIDENT) {
#pragma unroll
    for (int k = 0; k < OWN; ++k) x[k] = r[k] = m[k] = 0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) p[d] = y[d] = 0;
    if (mine) {
      row = rows_own<DIM>(A, s, P.x, p);
      if (P.warm) rows_product<DIM, WIDE>(A, s, row, P.x, p, y);
      own_of(p, x);
      own_of(y, yo);
      NodeV<double, VW> f = ldv<double, VW>(P.f, row < 0 ? 0 : row), di = ldv<double, VW>(P.dinv, row < 0 ? 0 : row);
      double fa[DIM], fo[OWN], po[OWN];
#pragma unroll
      for (int d = 0; d < DIM; ++d) fa[d] = row < 0 ? 0.0 : f.v[d];
      own_of(fa, fo);
#pragma unroll
      for (int d = 0; d < DIM; ++d) fa[d] = row < 0 ? 0.0 : di.v[d];
      own_of(fa, m);
#pragma unroll
      for (int k = 0; k < OWN; ++k) {
        if (!P.warm || row < 0) x[k] = 0;
        r[k] = P.warm && row >= 0 ? fo[k] - yo[k] : fo[k];
        po[k] = r[k] * m[k];
        sums[0] += r[k] * po[k];
        sums[1] += r[k] * r[k];
        sums[2] += fo[k] * fo[k];
      }
      share_p(po);
      store_p();
    }
  } else {
    if (P.warm) {
      for (int64_t q = s0 + wid; q < s1; q += WARPS) {
        double xi[DIM], v[DIM];
        const int i = rows_own<DIM>(A, q, P.x, xi);
        rows_product<DIM, WIDE>(A, q, i, P.x, xi, v);
        if (i >= 0 && !half) {
          NodeV<double, VW> o;
#pragma unroll
          for (int d = 0; d < VW; ++d) o.v[d] = d < DIM ? v[d < DIM ? d : 0] : 0.0;
          stv<double, VW>(P.u, i, o);
        }
      }
      __syncthreads();
    }
    each_node([&](int n) {
      const NodeV<double, VW> f = ldv<double, VW>(P.f, n), di = ldv<double, VW>(P.dinv, n);
      NodeV<double, VW> u, rv, pv, zero;
#pragma unroll
      for (int d = 0; d < VW; ++d) zero.v[d] = u.v[d] = rv.v[d] = pv.v[d] = 0;
      if (P.warm) u = ldv<double, VW>(P.u, n);
      else stv<double, VW>(P.x, n, zero);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        rv.v[d] = P.warm ? f.v[d] - u.v[d] : f.v[d];
        pv.v[d] = rv.v[d] * di.v[d];
        sums[0] += rv.v[d] * pv.v[d];
        sums[1] += rv.v[d] * rv.v[d];
        sums[2] += f.v[d] * f.v[d];
      }
      stv<double, VW>(P.r, n, rv);
      stv<double, VW>(P.p, n, pv);
    });
  }
  // sqrt(rr) <= tol sqrt(ff) is tested as rr <= (tol sqrt(ff))^2
  if (!grid_sums<3>(G, 0, sums, sh, [&](const double (&t)[3]) {
        const double lim = tol * sqrt(t[2]);
        sh.total[kMaxGridSums] = lim < 0 ? -1.0 : lim * lim;  // (a negative tol stops nothing)
      }))
    return stalled();
  const double gamma0 = sums[0], ff = sums[2], rr_stop = sh.total[kMaxGridSums], gamma_stop = tol * gamma0;
  double gamma = gamma0, gamma_prev = gamma0, rr = sums[1], sigma = 0, alpha = 0, beta = 0;
  int it = 0, done = 0;
  if (gamma0 == 0.0) done = 1;
  if (rule == 1 && rr <= rr_stop) done = 1;
  if (!isfinite(gamma0)) done = 2;
  if (!grid_barrier(G, ++epoch, sh)) return stalled();
  while (!done) {
    const int set = 1 + 2 * (it & 1);
    double e[1] = {0};
    if constexpr (RESIDENT) {
      if (mine) {
        rows_product<DIM, WIDE>(A, s, row, P.p, p, y);
        double po[OWN];
        own_of(y, yo);
        own_of(p, po);
        if (row >= 0)
#pragma unroll
          for (int k = 0; k < OWN; ++k) e[0] += po[k] * yo[k];
      }
    } else {
      for (int64_t q = s0 + wid; q < s1; q += WARPS) {
        double pi[DIM], v[DIM];
        const int i = rows_own<DIM>(A, q, P.p, pi);
        rows_product<DIM, WIDE>(A, q, i, P.p, pi, v);
        if (i >= 0 && !half) {
          NodeV<double, VW> o;
#pragma unroll
          for (int d = 0; d < VW; ++d) o.v[d] = d < DIM ? v[d < DIM ? d : 0] : 0.0;
          stv<double, VW>(P.u, i, o);
#pragma unroll
          for (int d = 0; d < DIM; ++d) e[0] += pi[d] * v[d];
        }
      }
    }
    if (!grid_sums<1>(G, set, e, sh, [&](const double (&t)[1]) { sh.total[kMaxGridSums] = gamma / t[0]; }))
      return stalled();
    sigma = e[0];
    alpha = sh.total[kMaxGridSums];
    grid_reset<1>(G, 4 - set);  // (the sets of the next iteration)
    grid_reset<2>(G, 5 - set);
    double g[2] = {0, 0};
    if constexpr (RESIDENT) {
      if (mine) {
#pragma unroll
        for (int k = 0; k < OWN; ++k) {
          r[k] -= alpha * yo[k];
          const double z = r[k] * m[k];
          g[0] += r[k] * z;
          g[1] += r[k] * r[k];
        }
        if (row < 0) g[0] = g[1] = 0;
      }
    } else {
      each_node([&](int n) {
        NodeV<double, VW> rv = ldv<double, VW>(P.r, n), zv;
        const NodeV<double, VW> u = ldv<double, VW>(P.u, n), di = ldv<double, VW>(P.dinv, n);
#pragma unroll
        for (int d = 0; d < VW; ++d) zv.v[d] = 0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          rv.v[d] -= alpha * u.v[d];
          zv.v[d] = rv.v[d] * di.v[d];
          g[0] += rv.v[d] * zv.v[d];
          g[1] += rv.v[d] * rv.v[d];
        }
        stv<double, VW>(P.r, n, rv);
        stv<double, VW>(P.z, n, zv);
      });
    }
    if (!grid_sums<2>(G, set + 1, g, sh, [&](const double (&t)[2]) { sh.total[kMaxGridSums] = t[0] / gamma; }))
      return stalled();
    gamma_prev = gamma;
    gamma = g[0];
    rr = g[1];
    beta = sh.total[kMaxGridSums];
    ++it;
    if (!isfinite(gamma) || !isfinite(alpha)) done = 2;
    else if (rule == 0 && gamma < gamma_stop) done = 1;
    else if (rule == 1 && rr <= rr_stop) done = 1;
    else if (it >= maxit) done = 3;
    if constexpr (RESIDENT) {
      if (mine) {
        double po[OWN];
        own_of(p, po);
#pragma unroll
        for (int k = 0; k < OWN; ++k) {
          x[k] += alpha * po[k];
          po[k] = r[k] * m[k] + beta * po[k];
        }
        share_p(po);
        if (!done) store_p();
      }
    } else {
      each_node([&](int n) {  // (the last pass too: x of the step just taken)
        NodeV<double, VW> xv = ldv<double, VW>(P.x, n), pv = ldv<double, VW>(P.p, n);
        const NodeV<double, VW> zv = ldv<double, VW>(P.z, n);
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          xv.v[d] += alpha * pv.v[d];
          pv.v[d] = zv.v[d] + beta * pv.v[d];
        }
        stv<double, VW>(P.x, n, xv);
        if (!done) stv<double, VW>(P.p, n, pv);
      });
    }
    if (done) break;
    if (!grid_barrier(G, ++epoch, sh)) return stalled();
  }
  if constexpr (RESIDENT) {
    if (mine && row >= 0)
#pragma unroll
      for (int k = 0; k < OWN; ++k)
        if (c0 + k < DIM) P.x[(int64_t)row * VW + c0 + k] = x[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    Scalars *o = P.sc;
    o->gamma0 = gamma0;
    o->gamma = gamma;
    o->gamma_prev = gamma_prev;
    o->rr = rr;
    o->ff = ff;
    o->sigma = sigma;
    o->alpha = alpha;
    o->beta = beta;
    o->iter = it;
    o->done = done;
  }
}

// ------------------------------------------------------------------ construction
// Elements of every node (sorted), neighbour lists, slices, blocks.
static __global__ void k_rows_count(int64_t n, const int32_t *conn, int32_t *cnt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(cnt + conn[i], 1);
}

// out[0] = 0, out[i + 1] = in[0] + .. + in[i], one block of 1024 threads.
template <typename TO>
__global__ void __launch_bounds__(1024) k_rows_scan(int64_t n, const int32_t *in, TO *out) {
  __shared__ long long warp_sum[32];
  __shared__ long long carry_s;
  if (threadIdx.x == 0) {
    carry_s = 0;
    out[0] = 0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t base = 0; base < n; base += 4096) {
    long long v[4], t = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = base + threadIdx.x * 4 + q;
      t += i < n ? in[i] : 0;
      v[q] = t;
    }
    long long inc = t;
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) warp_sum[wid] = inc;
    __syncthreads();
    if (wid == 0) {
      long long w = warp_sum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    const long long before = carry_s + (wid ? warp_sum[wid - 1] : 0) + inc - t;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = base + threadIdx.x * 4 + q;
      if (i < n) out[i + 1] = (TO)(before + v[q]);
    }
    __syncthreads();
    if (threadIdx.x == 0) carry_s += warp_sum[31];
    __syncthreads();
  }
}

static __global__ void k_rows_fill(int64_t n, int nv, const int32_t *conn, const int32_t *inc_off, int32_t *cursor,
                                   int32_t *inc) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t v = conn[i];
  inc[inc_off[v] + atomicAdd(cursor + v, 1)] = (int32_t)(i / nv);
}

// ascending in-place sort of one thread's list: insertion while short, heap sort beyond
__device__ __forceinline__ void sort_list(int32_t *a, int n) {
  if (n <= 96) {
    for (int i = 1; i < n; ++i) {
      const int32_t v = a[i];
      int j = i;
      for (; j > 0 && a[j - 1] > v; --j) a[j] = a[j - 1];
      a[j] = v;
    }
    return;
  }
  for (int start = n / 2 - 1, end = n; end > 1;) {
    int root;
    if (start >= 0) {
      root = start--;
    } else {
      --end;
      const int32_t t = a[end];
      a[end] = a[0];
      a[0] = t;
      root = 0;
    }
    for (int child; (child = 2 * root + 1) < end; root = child) {
      if (child + 1 < end && a[child + 1] > a[child]) ++child;
      if (a[root] >= a[child]) break;
      const int32_t t = a[root];
      a[root] = a[child];
      a[child] = t;
    }
  }
}

// One thread per node (blocks of one warp: the lists of 256 nodes do not stay in an
// L1): its elements sorted, its neighbours sorted and unique
// in nbr[(NV - 1) * inc_off[n] ..], their number in deg.
// n_wide: nodes of more than kWideDegree neighbours are counted.
template <int NV>
__global__ void k_rows_neighbours(int64_t nn, const int32_t *conn, const int32_t *inc_off, int32_t *inc, int32_t *nbr,
                                  int32_t *deg, int32_t *n_wide) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= nn) return;
  const int32_t i0 = inc_off[n], m = inc_off[n + 1] - i0;
  sort_list(inc + i0, m);
  int32_t *list = nbr + (int64_t)(NV - 1) * i0;
  int c = 0;
  if ((NV - 1) * m <= 96) {  // insert, skipping what is there
    for (int q = 0; q < m; ++q)
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        const int32_t v = conn[(int64_t)inc[i0 + q] * NV + a];
        if (v == n) continue;
        int j = c;
        for (; j > 0 && list[j - 1] > v; --j) {}
        if (j > 0 && list[j - 1] == v) continue;
        for (int t = c; t > j; --t) list[t] = list[t - 1];
        list[j] = v;
        ++c;
      }
  } else {
    for (int q = 0; q < m; ++q)
      for (int a = 0; a < NV; ++a) {
        const int32_t v = conn[(int64_t)inc[i0 + q] * NV + a];
        if (v != n) list[c++] = v;
      }
    sort_list(list, c);
    int u = 0;
    for (int t = 0; t < c; ++t)
      if (t == 0 || list[t] != list[t - 1]) list[u++] = list[t];
    c = u;
  }
  deg[n] = c;
  if (c > kWideDegree) atomicAdd(n_wide, 1);
}

// Rows of each window by descending neighbour count (ties by node), and the
// steps of each slice. One block per window.
static __global__ void __launch_bounds__(kRowWindow) k_rows_order(int64_t nn, const int32_t *deg, int32_t *row,
                                                                  int32_t *steps) {
  __shared__ int32_t d[kRowWindow];
  const int64_t base = (int64_t)blockIdx.x * kRowWindow;
  const int t = threadIdx.x, n = (int)min((int64_t)kRowWindow, nn - base);
  d[t] = t < n ? deg[base + t] : -1;
  __syncthreads();
  const int mine = d[t];
  int rank = 0;
  for (int j = 0; j < kRowWindow; ++j) rank += d[j] > mine || (d[j] == mine && j < t);
  row[base + rank] = t < n ? (int32_t)(base + t) : -1;
  if (rank % kSliceRows == 0) steps[(base + rank) / kSliceRows] = mine < 0 ? 0 : (mine + 1) / 2;
}

// The same where there are nodes of many neighbours: they come first in their
// window's slices, one in each. First the slices of every window, then rows (-1 at
// the start) and steps, with `first` the windows' first slices.
static __global__ void __launch_bounds__(kRowWindow) k_rows_window_slices(int64_t nn, const int32_t *deg, int32_t *slices) {
  const int64_t i = (int64_t)blockIdx.x * kRowWindow + threadIdx.x;
  const int wide = __syncthreads_count(i < nn && deg[i] > kWideDegree);
  const int n = (int)min((int64_t)kRowWindow, nn - (int64_t)blockIdx.x * kRowWindow);
  if (threadIdx.x == 0) slices[blockIdx.x] = wide + (n - wide + kSliceRows - 1) / kSliceRows;
}
static __global__ void __launch_bounds__(kRowWindow)
    k_rows_order_wide(int64_t nn, const int32_t *deg, const int32_t *first, int32_t *row, int32_t *steps, uint8_t *wide) {
  __shared__ int32_t d[kRowWindow];
  const int64_t base = (int64_t)blockIdx.x * kRowWindow;
  const int t = threadIdx.x, n = (int)min((int64_t)kRowWindow, nn - base);
  const int mine = t < n ? deg[base + t] : -1;
  d[t] = mine;
  const int n_wide = __syncthreads_count(mine > kWideDegree);
  if (t >= n) return;
  int rank = 0;
  for (int j = 0; j < kRowWindow; ++j) rank += d[j] > mine || (d[j] == mine && j < t);
  const bool own = rank < n_wide;
  const int q = rank - n_wide, s = first[blockIdx.x] + (own ? rank : n_wide + q / kSliceRows), at = own ? 0 : q % kSliceRows;
  row[(int64_t)s * kSliceRows + at] = (int32_t)(base + t);
  if (at == 0) {
    steps[s] = own ? (mine + 31) / 32 : (mine + 1) / 2;
    wide[s] = own ? kWideSlice : 0;
  }
}

// P_i K_ij P_j of the pair from the elements that hold both (in element order,
// so K_ij and K_ji are the same numbers), plus the consistent mass if cM != 0.
template <int DIM>
struct RowsAssembly {
  const int32_t *conn, *inc_off, *inc;
  const double *G64;
  int64_t gstride;
  double lam, mu, cK, cM;
  const double *lam_e, *mu_e;  // per-element material (new order) or nullptr
  const double *mc;            // per-element consistent-mass coefficient (cM != 0)
  const uint8_t *bits;
};

template <int DIM>
__device__ __forceinline__ void vertex_gradient(const RowsAssembly<DIM> &P, int64_t e, int a, double (&g)[DIM]) {
#pragma unroll
  for (int d = 0; d < DIM; ++d) g[d] = 0;
  if (a > 0) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) g[d] = P.G64[(size_t)((a - 1) * DIM + d) * P.gstride + e];
  } else {
#pragma unroll
    for (int b = 0; b < DIM; ++b)
#pragma unroll
      for (int d = 0; d < DIM; ++d) g[d] -= P.G64[(size_t)(b * DIM + d) * P.gstride + e];
  }
}

// The elements that a pair's block is looked for in: those of the node with fewer
// (a node of ten thousand elements costs its neighbours no more than their own
// lists), the same for (i, j) and (j, i).
template <int DIM>
__device__ __forceinline__ void pair_list(const RowsAssembly<DIM> &P, int32_t i, int32_t j, int32_t &q0, int32_t &q1) {
  q0 = P.inc_off[i];
  q1 = P.inc_off[i + 1];
  const int32_t r0 = P.inc_off[j], r1 = P.inc_off[j + 1];
  if (r1 - r0 < q1 - q0 || (r1 - r0 == q1 - q0 && j < i)) {
    q0 = r0;
    q1 = r1;
  }
}

// The unmasked block of the pair (i, j) from the elements inc[q], q0 <= q < q1, in
// steps of `step`, that hold both.
template <int DIM>
__device__ __forceinline__ void pair_block(const RowsAssembly<DIM> &P, int32_t i, int32_t j, int32_t q, int32_t q1,
                                           int step, double (&K)[DIM * DIM], double &mass) {
  constexpr int NV = DIM + 1;
#pragma unroll
  for (int c = 0; c < DIM * DIM; ++c) K[c] = 0;
  mass = 0;
  while (q < q1) {
    // elements holding j are collected first: the FP64 part then runs with
    // full warps
    int32_t hit[8];
    uint8_t at[8];
    int n = 0;
    for (; q < q1 && n < 8; q += step) {
      const int32_t e = P.inc[q];
      int ai = -1, aj = -1;
#pragma unroll
      for (int a = 0; a < NV; ++a) {
        const int32_t v = P.conn[(int64_t)e * NV + a];
        if (v == i) ai = a;
        if (v == j) aj = a;
      }
      if (ai >= 0 && aj >= 0) {
        hit[n] = e;
        at[n] = (uint8_t)(ai * 4 + aj);
        ++n;
      }
    }
    for (int t = 0; t < n; ++t) {
      const int64_t e = hit[t];
      double gi[DIM], gj[DIM], dot = 0;
      vertex_gradient<DIM>(P, e, at[t] >> 2, gi);
      vertex_gradient<DIM>(P, e, at[t] & 3, gj);
#pragma unroll
      for (int d = 0; d < DIM; ++d) dot += gi[d] * gj[d];
      const double lam = P.lam_e ? P.lam_e[e] : P.lam, mu = P.mu_e ? P.mu_e[e] : P.mu;
#pragma unroll
      for (int p = 0; p < DIM; ++p)
#pragma unroll
        for (int r = 0; r < DIM; ++r)
          K[p * DIM + r] += lam * (gi[p] * gj[r]) + mu * (gi[r] * gj[p]) + (p == r ? mu * dot : 0.0);
      if (P.cM != 0) mass += P.mc[e];
    }
  }
}

// Columns (first assembly) and blocks, eight warps per slice: a step is a chain of
// dependent loads (lists, elements, gradients), so the steps of a slice side by
// side are what a small mesh has to fill the GPU with. Whole cfem_set_young, one
// warp per slice and so: 12,288 tets 0.42 -> 0.18 ms, 98,304 0.54 -> 0.36,
// 2.65 M 5.73 -> 5.6, 130,000 Delaunay tets 1.50 -> 0.59. (Four warps, and eight
// lanes per row of the corrections below: 0.20, 0.38, 5.55, 0.64.)
constexpr int kAssembleWarps = 8;
constexpr int kLongList = 64;  // elements that one lane goes through alone
template <int DIM>
__global__ void __launch_bounds__(32 * kAssembleWarps) k_rows_assemble(RowsAssembly<DIM> P, const int64_t *off,
                                                       const int32_t *row, const int32_t *nbr, const int32_t *deg,
                                                       int32_t *col, double *val, const uint8_t *flag) {
  constexpr int NC = DIM * DIM, NV = DIM + 1;
  const int64_t s = blockIdx.x;
  const bool wide = flag[s] & kWideSlice;
  const int lane = threadIdx.x & 31;
  const int32_t i = row[s * kSliceRows + (wide ? 0 : lane & 15)];
  const int64_t k0 = off[s];
  const int n = (int)(off[s + 1] - k0);
  const unsigned bi = i < 0 ? 0u : P.bits[i];
  for (int k = threadIdx.x >> 5; k < n; k += kAssembleWarps) {
    const int64_t at = (k0 + k) * 32 + lane;
    int32_t j;
    if (nbr) {  // first assembly: the columns from the neighbour lists
      j = i < 0 ? 0 : i;
      const int at_i = wide ? 32 * k + lane : 2 * k + (lane >> 4);
      if (i >= 0 && at_i < deg[i]) j = nbr[(int64_t)(NV - 1) * P.inc_off[i] + at_i];
      col[at] = j;
    } else {
      j = col[at];
    }
    double K[NC], m = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) K[c] = 0;
    int32_t q0 = 0, q1 = 0;
    if (i >= 0 && j != i) pair_list<DIM>(P, i, j, q0, q1);
    const bool long_list = q1 - q0 > kLongList;
    if (q0 < q1 && !long_list) pair_block<DIM>(P, i, j, q0, q1, 1, K, m);
    // (an edge that many elements share: the warp goes through them together)
    for (unsigned todo = __ballot_sync(0xffffffffu, long_list); todo; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const int32_t ii = __shfl_sync(0xffffffffu, i, src), jj = __shfl_sync(0xffffffffu, j, src);
      const int32_t a = __shfl_sync(0xffffffffu, q0, src), b = __shfl_sync(0xffffffffu, q1, src);
      double S[NC], sm;
      pair_block<DIM>(P, ii, jj, a + lane, b, 32, S, sm);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < NC; ++c) S[c] += __shfl_xor_sync(0xffffffffu, S[c], o);
        sm += __shfl_xor_sync(0xffffffffu, sm, o);
      }
      if (lane == src) {
#pragma unroll
        for (int c = 0; c < NC; ++c) K[c] = S[c];
        m = sm;
      }
    }
    const unsigned bj = i < 0 ? 0u : P.bits[j];
    double *v = val + (k0 + k) * (32 * NC) + lane;
#pragma unroll
    for (int p = 0; p < DIM; ++p)
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        double t = P.cK * K[p * DIM + q];
        if (p == q && P.cM != 0) t += P.cM * m;
        v[(p * DIM + q) * 32] = ((bi >> p) & 1u) || ((bj >> q) & 1u) ? 0.0 : t;
      }
  }
}

// D blocks: what the difference form misses (see the head of this file), sixteen
// lanes per row, which share its neighbours and elements; a slice with any is
// flagged.
constexpr int kCorrLanes = 16;
template <int DIM>
__global__ void k_rows_corrections(RowsAssembly<DIM> P, int64_t n_rows, const int64_t *off, const int32_t *row,
                                   const int32_t *col, double *D, uint8_t *flag) {
  constexpr int NC = DIM * DIM;
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kCorrLanes;
  const int part = threadIdx.x % kCorrLanes;
  const int32_t i = t < n_rows ? row[t] : -1;
  const int64_t s = t / kSliceRows;
  const unsigned bi = i < 0 ? 0u : P.bits[i];
  double B[NC], diag[DIM], mass = 0;
#pragma unroll
  for (int c = 0; c < NC; ++c) B[c] = 0;
#pragma unroll
  for (int p = 0; p < DIM; ++p) diag[p] = 0;
  bool any = i >= 0 && (bi != 0 || P.cM != 0);
  const bool wide = i >= 0 && (flag[s] & kWideSlice);
  const int width = wide ? 1 : 16;  // entries q of the row are this far apart
  if (i >= 0)
    for (int64_t q = 32 / width * off[s] + part; q < 32 / width * off[s + 1]; q += kCorrLanes) {
      const int32_t j = col[q * width + (t & 15)];
      if (j == i) continue;
      const unsigned bj = P.bits[j];
      if (bj == bi && P.cM == 0) continue;
      any = true;
      double K[NC], m;
      int32_t e0, e1;
      pair_list<DIM>(P, i, j, e0, e1);
      pair_block<DIM>(P, i, j, e0, e1, 1, K, m);
#pragma unroll
      for (int p = 0; p < DIM; ++p)
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          const int fj = !((bj >> r) & 1u), fi = !((bi >> r) & 1u);
          B[p * DIM + r] += P.cK * K[p * DIM + r] * (double)(fj - fi);
          // mass: M_ij x_j = M_ij (x_j - x_i) + M_ij x_i on free DOFs
          if (p == r) B[p * DIM + r] += P.cM * m * (double)fj;
        }
    }
  if (!__any_sync(0xffffffffu, any)) {
    if (i >= 0)
      for (int c = part; c < NC; c += kCorrLanes) D[(int64_t)i * NC + c] = 0.0;
    return;
  }
  // mass, and the diagonal of constrained DOFs, from the node's elements
  if (i >= 0 && (bi || P.cM != 0))
    for (int32_t q = P.inc_off[i] + part; q < P.inc_off[i + 1]; q += kCorrLanes) {
      const int32_t e = P.inc[q];
      if (P.cM != 0) mass += 2.0 * P.mc[e];  // M_ii = twice the element coefficients
      if (!bi) continue;
      int a = 0;
#pragma unroll
      for (int v = 1; v <= DIM; ++v)
        if (P.conn[(int64_t)e * (DIM + 1) + v] == i) a = v;
      double g[DIM], tot = 0;
      vertex_gradient<DIM>(P, e, a, g);
      const double lam = P.lam_e ? P.lam_e[e] : P.lam, mu = P.mu_e ? P.mu_e[e] : P.mu;
#pragma unroll
      for (int p = 0; p < DIM; ++p) tot += g[p] * g[p];
#pragma unroll
      for (int p = 0; p < DIM; ++p) diag[p] += (lam + 2 * mu) * (g[p] * g[p]) + mu * (tot - g[p] * g[p]);
    }
#pragma unroll
  for (int o = kCorrLanes / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) B[c] += __shfl_xor_sync(0xffffffffu, B[c], o);
#pragma unroll
    for (int p = 0; p < DIM; ++p) diag[p] += __shfl_xor_sync(0xffffffffu, diag[p], o);
    mass += __shfl_xor_sync(0xffffffffu, mass, o);
  }
  if (i < 0) return;
#pragma unroll
  for (int p = 0; p < DIM; ++p) {
    B[p * DIM + p] += P.cM * mass;
    if ((bi >> p) & 1u)  // constrained: the diagonal of cK K + cM M alone
#pragma unroll
      for (int r = 0; r < DIM; ++r) B[p * DIM + r] = p == r ? P.cK * diag[p] + P.cM * mass : 0.0;
  }
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (c % kCorrLanes == part) D[(int64_t)i * NC + c] = B[c];
  if (any) flag[s] = wide ? kWideSlice | kHasD : kHasD;  // (the same from every lane)
}

}  // namespace cfem
