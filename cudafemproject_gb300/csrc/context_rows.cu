// Host side of the FP64 row operator (kernels_rows.cuh): construction when a
// context is created or its moduli change, applications, true residuals.
#include "context_internal.cuh"
#include "kernels_aux.cuh"
#include "rows_op.cuh"

namespace cfem {
namespace detail {

namespace {

template <int DIM>
RowsAssembly<DIM> assembly(cfem_ctx *c, double cK, double cM) {
  RowsAssembly<DIM> P{};
  P.conn = c->conn.p;
  P.inc_off = c->rows.inc_off.p;
  P.inc = c->rows.inc.p;
  P.G64 = c->G64.p;
  P.gstride = c->gstride;
  P.lam = c->lam;
  P.mu = c->mu;
  P.cK = cK;
  P.cM = cM;
  P.lam_e = c->lam_e.p;
  P.mu_e = c->mu_e.p;
  P.mc = c->mc64.p;
  P.bits = c->bits.p;
  return P;
}

// Node-element incidences, neighbour lists, row order and slices; the
// neighbour lists stay in `nbr` for the first assembly.
template <int NV>
void build_structure(cfem_ctx *c, DBuf<int32_t> &nbr, DBuf<int32_t> &deg) {
  RowsData &R = c->rows;
  cudaStream_t s = c->stream;
  const int64_t nn = c->nn, n_inc = c->ne * NV;
  const int64_t windows = (nn + kRowWindow - 1) / kRowWindow, n_steps = windows * (kRowWindow / kSliceRows);
  R.n_slices = (nn + kSliceRows - 1) / kSliceRows;  // (the padding sorts last)
  // what stays, in one allocation: inc_off, inc, row (off: 8-byte aligned first)
  auto even = [](int64_t n) { return (n + 3) / 4 * 4; };
  R.slab.alloc((size_t)(2 * even(R.n_slices + 1) + even(nn + 1) + even(n_inc) + even(windows * kRowWindow)));
  int32_t *at = R.slab.p;
  R.off.view(reinterpret_cast<int64_t *>(at), R.n_slices + 1);
  at += 2 * even(R.n_slices + 1);
  R.inc_off.view(at, nn + 1);
  at += even(nn + 1);
  R.inc.view(at, n_inc);
  at += even(n_inc);
  R.row.view(at, (size_t)windows * kRowWindow);
  // what the construction needs: neighbour lists, their lengths, counts, steps per slice
  nbr.alloc((size_t)(even((NV - 1) * n_inc) + 2 * even(nn) + n_steps + 1));
  int32_t *deg_p = nbr.p + even((NV - 1) * n_inc), *cnt = deg_p + even(nn), *steps = cnt + even(nn);
  int32_t *n_wide = steps + n_steps, *h_wide = reinterpret_cast<int32_t *>(c->h_rr + 1);
  CK(cudaMemsetAsync(n_wide, 0, sizeof(int32_t), s));
  deg.view(deg_p, nn);
  CK(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * nn, s));
  k_rows_count<<<nblk(n_inc), kThreads, 0, s>>>(n_inc, c->conn.p, cnt);
  k_rows_scan<int32_t><<<1, 1024, 0, s>>>(nn, cnt, R.inc_off.p);
  CK(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * nn, s));
  k_rows_fill<<<nblk(n_inc), kThreads, 0, s>>>(n_inc, NV, c->conn.p, R.inc_off.p, cnt, R.inc.p);
  k_rows_neighbours<NV><<<nblk(nn, 32), 32, 0, s>>>(nn, c->conn.p, R.inc_off.p, R.inc.p, nbr.p, deg.p, n_wide);
  k_rows_order<<<(unsigned)windows, kRowWindow, 0, s>>>(nn, deg.p, R.row.p, steps);
  k_rows_scan<int64_t><<<1, 1024, 0, s>>>(R.n_slices, steps, R.off.p);
  CKL();
  CK(cudaMemcpyAsync(c->h_rr, R.off.p + R.n_slices, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(h_wide, n_wide, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (*(volatile int32_t *)h_wide) {  // slices of one row for the nodes of many neighbours
    DBuf<int32_t> first;  // slices of each window, their first ones, steps of each slice
    first.alloc((size_t)(2 * windows + 1));
    k_rows_window_slices<<<(unsigned)windows, kRowWindow, 0, s>>>(nn, deg.p, first.p);
    k_rows_scan<int32_t><<<1, 1024, 0, s>>>(windows, first.p, first.p + windows);
    CKL();
    CK(cudaMemcpyAsync(h_wide, first.p + 2 * windows, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    R.n_slices = *(volatile int32_t *)h_wide;
    R.off.alloc(R.n_slices + 1);
    R.row.alloc((size_t)R.n_slices * kSliceRows);
    R.wide.alloc(R.n_slices);
    DBuf<int32_t> steps_of;
    steps_of.alloc(R.n_slices);
    CK(cudaMemsetAsync(R.row.p, 0xFF, sizeof(int32_t) * R.row.n, s));
    k_rows_order_wide<<<(unsigned)windows, kRowWindow, 0, s>>>(nn, deg.p, first.p + windows, R.row.p, steps_of.p, R.wide.p);
    k_rows_scan<int64_t><<<1, 1024, 0, s>>>(R.n_slices, steps_of.p, R.off.p);
    CKL();
    CK(cudaMemcpyAsync(c->h_rr, R.off.p + R.n_slices, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
  }
  R.steps = *(volatile int64_t *)c->h_rr;
  R.col.alloc((size_t)R.steps * 32);
}

template <int DIM>
void assemble_dim(cfem_ctx *c, const int32_t *nbr, const int32_t *deg, double cK, double cM, RowsValues &V) {
  RowsData &R = c->rows;
  cudaStream_t s = c->stream;
  if (!V.val.p) {
    const size_t n_val = (size_t)R.steps * 32 * DIM * DIM, n_D = (size_t)c->nn * DIM * DIM;
    V.val.alloc(n_val + n_D + (R.n_slices + 7) / 8);
    V.D.view(V.val.p + n_val, n_D);
    V.flag.view(reinterpret_cast<uint8_t *>(V.val.p + n_val + n_D), R.n_slices);
  }
  if (R.wide.p) CK(cudaMemcpyAsync(V.flag.p, R.wide.p, R.n_slices, cudaMemcpyDeviceToDevice, s));
  else V.flag.zero(s);
  const RowsAssembly<DIM> P = assembly<DIM>(c, cK, cM);
  k_rows_assemble<DIM><<<(unsigned)R.n_slices, 32 * kAssembleWarps, 0, s>>>(P, R.off.p, R.row.p, nbr, deg, R.col.p,
                                                            V.val.p, V.flag.p);
  k_rows_corrections<DIM><<<nblk(R.n_slices * kSliceRows * kCorrLanes), kThreads, 0, s>>>(P, R.n_slices * kSliceRows, R.off.p,
                                                                             R.row.p, R.col.p, V.D.p, V.flag.p);
  CKL();
}

void assemble(cfem_ctx *c, const int32_t *nbr, const int32_t *deg, double cK, double cM, RowsValues &V) {
  if (c->dim == 3) assemble_dim<3>(c, nbr, deg, cK, cM, V);
  else assemble_dim<2>(c, nbr, deg, cK, cM, V);
}

unsigned rows_grid(const cfem_ctx *c) { return nblk(c->rows.n_slices, kRowsThreads / 32); }

}  // namespace

RowOp op_of(cfem_ctx *c, const RowsValues &V) {
  const RowsData &R = c->rows;
  return RowOp{R.n_slices, R.off.p, R.row.p, R.col.p, V.val.p, V.flag.p, V.D.p, c->bits.p};
}

GridSync start_grid_sync(cfem_ctx *c, int sets) {
  const size_t n = grid_slots_count(kRowsPcgSets, c->n_sm);
  if (!c->grid_slots.p) c->grid_slots.alloc(n + 1);  // (the barrier's counter follows the slots)
  if (sets) CK(cudaMemsetAsync(c->grid_slots.p, 0xFF, n * sizeof(unsigned long long), c->stream));
  CK(cudaMemsetAsync(c->grid_slots.p + n, 0, sizeof(unsigned long long), c->stream));
  GridSync G{c->grid_slots.p, reinterpret_cast<unsigned *>(c->grid_slots.p + n), kWaitCycles, 0};
  if (c->selftest_absent && --c->selftest_absent == 0) {
    G.limit = 2000000;
    G.absent_plus1 = 1;
  }
  return G;
}

void build_rows(cfem_ctx *c) {
  c->rows.km_cK = c->rows.km_cM = -1;  // (combined values of an earlier operator are stale)
  if (!c->rows.col.p) {
    DBuf<int32_t> nbr, deg;
    if (c->dim == 3) build_structure<4>(c, nbr, deg);
    else build_structure<3>(c, nbr, deg);
    assemble(c, nbr.p, deg.p, 1.0, 0.0, c->rows.K);
    CK(cudaStreamSynchronize(c->stream));  // (before nbr is freed)
  } else {
    assemble(c, nullptr, nullptr, 1.0, 0.0, c->rows.K);
  }
}

void rows_apply(cfem_ctx *c, const double *x, double *y, bool caller_order) {
  const RowOp A = op_of(c, c->rows.K);
  auto go = [&](auto k) { k<<<rows_grid(c), kRowsThreads, 0, c->stream>>>(A, x, y, c->node_new2old.p); };
  auto pick = [&](auto wide) {
    constexpr bool W = decltype(wide)::value;
    if (c->dim == 3) caller_order ? go(k_rows_apply<3, true, W>) : go(k_rows_apply<3, false, W>);
    else caller_order ? go(k_rows_apply<2, true, W>) : go(k_rows_apply<2, false, W>);
  };
  if (c->rows.wide.p) pick(std::true_type{});
  else pick(std::false_type{});
  CKL();
  c->launches += 1;
}

// FP64 true residual r = f - K' x (f, x internal FP64; x == nullptr stands
// for x = 0), ||r||^2 and ||f||^2 into the device doubles out2[0], out2[1];
// queued on the context's stream.
void true_residual_async(cfem_ctx *c, const double *f, const double *x, double *r, float *r32, double *out2) {
  const RowOp A = op_of(c, c->rows.K);
  RowsResidual P{c->nn, f, x, r, r32, out2, c->partials.p, c->counters.p};
  // (grid-stride over the slices: the partial sums are one pair per block)
  const unsigned g = std::min<unsigned>(rows_grid(c), c->grid_rows);
  auto go = [&](auto k) { k<<<g, kRowsThreads, 0, c->stream>>>(A, P); };
  if (c->rows.wide.p) c->dim == 3 ? go(k_rows_residual<3, true>) : go(k_rows_residual<2, true>);
  else c->dim == 3 ? go(k_rows_residual<3, false>) : go(k_rows_residual<2, false>);
  CKL();
  c->launches += 1;
}

// FP64 Jacobi PCG on A x = V.f, A = cM M + cK K' (has_mass) or K', as one
// cooperative kernel (k_rows_pcg). V.dinv is the preconditioner; warm: V.x is
// the start.
PcgResult run_pcg_d(cfem_ctx *c, Vecs<double> &V, double cK, double cM, const double *mcoef, int warm, double tol,
                    int rule, int maxit) {
  RowsData &R = c->rows;
  const RowsValues *values = &R.K;
  if (mcoef || cK != 1.0) {  // implicit dynamics: stiffness and mass in the same blocks, assembled once per run
    if (!R.KM.val.p || R.km_cK != cK || R.km_cM != cM) {
      assemble(c, nullptr, nullptr, cK, mcoef ? cM : 0.0, R.KM);
      R.km_cK = cK;
      R.km_cM = cM;
    }
    values = &R.KM;
  }
  Scalars *sc = c->sc.p;
  Scalars h{};
  h.tol = tol;
  h.rule = rule;
  h.maxit = maxit > 0 ? maxit : 1000000;
  CK(cudaMemcpyAsync(sc, &h, sizeof(Scalars), cudaMemcpyHostToDevice, c->stream));
  RowsPcg P{};
  P.A = op_of(c, *values);
  P.f = V.f.p;
  P.dinv = V.dinv.p;
  P.x = V.x.p;
  P.r = V.r.p;
  P.z = V.z.p;
  P.p = V.pA.p;
  P.u = V.u.p;
  P.sc = sc;
  P.sync = start_grid_sync(c, kRowsPcgSets);
  P.warm = warm;
  // One CTA per SM, and fewer while a CTA has a quarter of an SM for each of
  // its slices: an exchange among 76 CTAs takes 0.4 us less than among 152, and
  // a slice runs no faster alone on an SM.
  const int grid = (int)std::min<int64_t>(c->n_sm, (R.n_slices + 3) / 4);
  const bool wide = R.wide.p;  // (one instance per dimension for every size: few meshes have such nodes)
  const bool small = !wide && R.n_slices <= (int64_t)grid * (kRowsPcgSmall / 32);
  const bool resident = R.n_slices <= (int64_t)grid * (kRowsPcgThreads / 32);
  auto pick = [&](auto k3, auto k2) { return c->dim == 3 ? (const void *)k3 : (const void *)k2; };
  const void *k = wide       ? pick(k_rows_pcg<3, false, kRowsPcgThreads, true>, k_rows_pcg<2, false, kRowsPcgThreads, true>)
                  : small    ? pick(k_rows_pcg<3, true, kRowsPcgSmall>, k_rows_pcg<2, true, kRowsPcgSmall>)
                  : resident ? pick(k_rows_pcg<3, true, kRowsPcgThreads>, k_rows_pcg<2, true, kRowsPcgThreads>)
                             : pick(k_rows_pcg<3, false, kRowsPcgThreads>, k_rows_pcg<2, false, kRowsPcgThreads>);
  void *args[] = {&P};
  CK(cudaLaunchCooperativeKernel(k, dim3(grid), dim3(small ? kRowsPcgSmall : kRowsPcgThreads), args, 0, c->stream));
  c->launches += 1;
  CK(cudaMemcpyAsync(c->h_sc, sc, sizeof(Scalars), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if (c->h_sc->stalled) throw Fail{CFEM_ERR_CUDA, "a CTA of the FP64 PCG kernel did not arrive at a grid-wide sum in time"};
  if (!c->h_sc->done) throw Fail{CFEM_ERR_CUDA, "PCG recurrence stopped advancing on the device"};
  if (c->verbose)
    std::printf("iteration %d gamma %.6e gamma0 %.6e\n", c->h_sc->iter, c->h_sc->gamma, c->h_sc->gamma0);
  PcgResult res;
  res.iters = c->h_sc->iter;
  res.gamma0 = c->h_sc->gamma0;
  res.gamma = c->h_sc->gamma;
  res.rr = c->h_sc->rr;
  res.ff = c->h_sc->ff;
  res.gamma_prev = c->h_sc->gamma_prev;
  const int d = c->h_sc->done;
  res.status = d == 1 ? CFEM_OK : d == 2 ? CFEM_ERR_DIVERGED : CFEM_ERR_NOT_CONVERGED;
  return res;
}

}  // namespace detail
}  // namespace cfem
