// Internals shared by the C-ABI translation units (context.cu, context_dyn.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "../../include/cfem.h"
#include "kernels.cuh"
#include "kernels_fan_tma.cuh"
#include "kernels_multi.cuh"
#include "kernels_batch.cuh"
#include "grid_sync.cuh"
#include "prep.hpp"

namespace cfem {
namespace detail {

extern thread_local std::string g_last_error;

struct MultiState;                    // multi-RHS work arrays (context_multi.cu)
void destroy_multi(MultiState *m);
struct BatchState;                    // batched solves (context_batch.cu)
void destroy_batch(BatchState *b);

struct Fail {
  cfem_status st;
  std::string msg;
};

#define CK(call)                                                                                   \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess)                                                                         \
      throw Fail{e_ == cudaErrorMemoryAllocation ? CFEM_ERR_OUT_OF_MEMORY : CFEM_ERR_CUDA,          \
                 std::string(#call) + ": " + cudaGetErrorString(e_)};                              \
  } while (0)

#define CKL() CK(cudaGetLastError())

template <typename T>
struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  bool owned = true;
  DBuf() = default;
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  ~DBuf() { release(); }
  void release() {
    if (p && owned) cudaFree(p);
    p = nullptr;
    n = 0;
    owned = true;
  }
  void view(T *at, size_t count) {  // part of a buffer that outlives this one
    release();
    p = at;
    n = count;
    owned = false;
  }
  void alloc(size_t count) {
    release();
    if (count == 0) return;
    CK(cudaMalloc(&p, count * sizeof(T)));
    n = count;
  }
  void ensure(size_t count) {  // at least count elements, contents undefined when it grows
    if (n < count) alloc(count);
  }
  void zero(cudaStream_t s) {
    if (p) CK(cudaMemsetAsync(p, 0, n * sizeof(T), s));
  }
  void upload(const T *h, size_t count, cudaStream_t s) {
    alloc(count);
    if (count) CK(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
  }
};

template <typename T>
struct Vecs {
  DBuf<T> slab;  // one allocation for all of them
  DBuf<T> x, r, z, pA, pB, u, uB, f, dinv, diagA;  // u, uB: A p of even, odd PCG iterations (FP32 only, like pB, diagA)
};

inline int pcg_chunk_from_env() {
  const char *e = std::getenv("CFEM_PCG_CHUNK");
  const int v = e ? std::atoi(e) : 16;
  return v < 2 ? 16 : (v + 1) & ~1;
}

struct GraphCache {
  cudaGraphExec_t exec = nullptr;
  bool device_loop = false;  // exec is a WHILE node around the iterations (one launch per solve)
  const void *key0 = nullptr;
  double key1 = 0, key2 = 0;
  int chunk = 0;  // iterations per body
  ~GraphCache() { reset(); }
  void reset() {
    if (exec) cudaGraphExecDestroy(exec);
    exec = nullptr;
  }
};

// FP64 operator as assembled node rows (kernels_rows.cuh): structure, and the
// values of one combination of stiffness and mass.
struct RowsValues {
  DBuf<double> val, D;
  DBuf<uint8_t> flag;
};
struct RowsData {
  DBuf<int32_t> slab;          // off, inc_off, inc, row
  DBuf<int32_t> inc_off, inc;  // elements of every node
  DBuf<int32_t> row, col;
  DBuf<int64_t> off;
  DBuf<uint8_t> wide;  // slices of one row (kWideSlice), or nothing
  int64_t n_slices = 0, steps = 0;
  RowsValues K;                 // stiffness
  RowsValues KM;                // km_cK K + km_cM M of the last implicit FP64 run
  double km_cK = -1, km_cM = -1;
};

// Work buffers of the time-stepping calls, kept with the context.
template <typename T>
struct StepVecs {
  DBuf<T> d, v, a, y, minv;  // d: two node vectors (three, FP32 implicit); v, a: two, y: three (FP32 fused steps); minv: two when re-sorted
};
struct StepWork {
  StepVecs<double> f64;
  StepVecs<float> f32;
  DBuf<double> coef, stress, diag_pre, diag_op, trace, obs, grad, young, states;
  DBuf<int32_t> recv, rec_head, rec_next;
  DBuf<DynState> st;
  DBuf<int> stalled;
  bool smem_raised = false;       // raise_smem_limit for the context's step kernel with re-sorted masses
  Scalars *ring = nullptr;        // pinned: scalars of the implicit steps in flight
  cudaEvent_t done[2] = {nullptr, nullptr};
  ~StepWork() {
    if (ring) cudaFreeHost(ring);
    for (cudaEvent_t e : done)
      if (e) cudaEventDestroy(e);
  }
};

inline unsigned nblk(int64_t n, int t = kThreads) { return (unsigned)((n + t - 1) / t); }

}  // namespace detail
}  // namespace cfem

using namespace cfem;
using namespace cfem::detail;

struct cfem_ctx {
  cudaStream_t stream = nullptr;       // the stream all work is issued on (capturable)
  cudaStream_t user_stream = nullptr;  // the caller's stream; work is ordered after it
  bool own_stream = false;
  cudaEvent_t ev_in = nullptr;
  int device = 0, n_sm = 0, l2_bytes = 0;
  int dim = 0, nv = 0, w = 0, vw = 0, ncomp = 0;
  int64_t nn = 0, ne = 0, nd = 0, nvec = 0;
  int semantics = 0, form = CFEM_FORM_GRADIENT, verbose = 0;
  double E = 0, nu = 0, rho = 0, lam = 0, mu = 0;
  Prep prep;
  RhsParts rhs;
  bool has_young = false;  // per-element moduli in young_d (caller order)
  double lump_c = 0, cons_c = 0;
  // mesh on device
  DBuf<int32_t> elem_off, node_off, nodes, own, node_new2old, elem_new2old, elem_old2new, conn;
  DBuf<uint2> lconn;
  DBuf<uint16_t> inc, inc_start;  // per-patch incidence lists
  // edge-fan form (3D): fan tables, gradients in fan vertex order
  bool fans = false;
  DBuf<int32_t> fan_off, fan_elem_off, fan_pos;
  DBuf<uint8_t> fan_perm;
  // edge-fan form, FP32, with bulk-copied patch blocks (kernels_fan_tma.cuh)
  FanBlockLayout L32{};
  DBuf<unsigned char> blk32;
  DBuf<int32_t> fan_patch;
  int *h_tma_err = nullptr;  // pinned; written by a kernel whose copy wait ran out
  int selftest_skip_plus1 = 0;       // FanTmaParams::skip_patch_plus1 (cfem_selftest_copy_timeout only)
  long long selftest_wait_limit = 0;  // FanTmaParams::wait_limit (likewise)
  int selftest_absent = 0;            // the n-th cooperative launch from here runs without its CTA 0 (cfem_selftest_grid_timeout only)
  size_t smem_ft32 = 0;
  int grid_ft32 = 0;
  // geometry blocks (FP32 single-RHS matvec of CFEM_FORM_GEOMETRY_FAN): the
  // prefix of blk32, then patch-relative coordinates and per-tet moduli scales
  bool geo = false;
  FanBlockLayout Lg{};
  DBuf<unsigned char> blkg;
  size_t smem_geo = 0;
  int grid_geo = 0;
  int np_slots = 0;               // node slots per patch in shared memory
  RowsData rows;                  // FP64 operator
  StepWork steps;
  DBuf<unsigned long long> grid_slots;  // grid-wide sums of the one-kernel PCG (grid_sync.cuh)
  int grid_rows = 0;              // CTAs of a grid-stride kernel over its slices
  DBuf<uint8_t> bits;
  DBuf<double> coords, escale, young_d;
  // operator
  int64_t gstride = 0;
  DBuf<double> G64, vol, diagK, mlump, mcdiag, mc64;
  DBuf<float> G32, mc32, diagK32;
  DBuf<double> FA, FB;
  DBuf<float> FA32, FB32;
  // work
  Vecs<double> v64;
  Vecs<float> v32;
  DBuf<double> io, tmp64, tmp64b;
  DBuf<Scalars> sc;  // [0] FP64 solve, [1] FP32 solve, [2] misc counters
  DBuf<double> partials;     // grid-sum scratch; the PCG-form matvec's p.Ap partials
  DBuf<double> partials_up;  // r.z, r.r partials of the PCG update kernel [grid][2]
  DBuf<unsigned int> counters;
  DBuf<int> err;
  void *pinned = nullptr;  // h_sc, h_rr, h_tma_err
  Scalars *h_sc = nullptr;
  double *h_rr = nullptr;
  int grid_mv = 0, grid_vec = 0;
  size_t smem64 = 0, smem32 = 0;
  // PCG iterations per graph body (even: the A p buffers alternate);
  // CFEM_PCG_CHUNK overrides it (rounded up to even)
  int chunk = pcg_chunk_from_env();
  // run the PCG iterations from the host, `chunk` per graph launch, instead of
  // inside a graph WHILE node (CFEM_HOST_LOOP set in the environment)
  bool host_loop = std::getenv("CFEM_HOST_LOOP") != nullptr;
  MultiState *multi = nullptr;
  BatchState *batch = nullptr;
  // batch of independent meshes (cfem_create_batch); n_inst == 0 for one mesh
  int n_inst = 0;
  std::vector<int32_t> elem_group;               // caller element -> instance
  std::vector<double> inst_lam, inst_mu;
  std::vector<int64_t> inst_node_off, inst_elem_off;  // caller order
  DBuf<int32_t> patch_inst, inst_patch_off, own_first;
  std::vector<int32_t> h_inst_patch_off, h_own_first;
  DBuf<float> pmat32;
  DBuf<double> lam_e, mu_e;
  int64_t launches = 0;  // kernels issued since the counter was last reset
  GraphCache graph32;
  bool diag_is_K = false;  // dinv and diagA of v64 and v32 belong to diagK
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // reference re-sorting quirk (compat dynamics)
  DBuf<int64_t> seg;
  DBuf<int32_t> perm, node_old2new;
  DBuf<double> slot_src, slot_tmp;

  ~cfem_ctx() {
    graph32.reset();
    if (pinned) cudaFreeHost(pinned);
    if (multi) destroy_multi(multi);
    if (batch) destroy_batch(batch);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (ev_in) cudaEventDestroy(ev_in);
    if (own_stream && stream) cudaStreamDestroy(stream);
  }
};


namespace cfem {
namespace detail {

// FP32_REFINE inner tolerances from which the inner PCG carries its search
// direction across the refinement steps (the tolerance is then the factor by
// which its recursive residual drops between FP64 true-residual replacements).
constexpr double kContinueTol = 0.2;
// A refinement step whose FP64 residual norm^2 falls by less than this is at
// the FP64 floor: a step cuts the norm by about the inner tolerance tol (at
// least halves it for tol up to 0.25), so the test allows twice that.
inline double refine_stall_ratio(double tol) { return std::min(0.9, std::max(0.25, 4.0 * tol * tol)); }

// Lets every launch of a kernel ask for as much dynamic shared memory as the
// device has beside its static part. The limit belongs to the kernel function and
// is shared by all contexts of the process, so it is only ever set to this one
// value: one of a context's own could be lowered by another thread's call between
// the setting and the launch.
inline void raise_smem_limit(const cfem_ctx *c, const void *kernel) {
  int optin = 0;
  cudaFuncAttributes at{};
  CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  CK(cudaFuncGetAttributes(&at, kernel));
  CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes));
}

// What a run of the FP32 PCG takes over from the one before: the last direction
// (p, nullptr: none) with the gamma its step length was formed with, and the last
// gamma (batched meshes: whether the recurrence still was the true residual).
struct PcgCont {
  const float *p = nullptr;
  double gamma_prev = 0, gamma = 0;
};

struct PcgResult {
  int status = CFEM_OK;
  int iters = 0;
  double gamma0 = 0, gamma = 0, rr = 0, ff = 0;
  double gamma_prev = 0;  // the gamma of the last step length (alpha = gamma_prev / p.Ap)
};

MvParams<double> base_mv_d(cfem_ctx *c);
MvParams<float> base_mv_f(cfem_ctx *c);
void launch_mv_f(cfem_ctx *c, int mode, const MvParams<float> &P);
PcgResult run_pcg_d(cfem_ctx *c, Vecs<double> &V, double cK, double cM, const double *mcoef, int warm, double tol,
                    int rule, int maxit);
PcgResult run_pcg_f(cfem_ctx *c, float cK, float cM, const float *mcoef, int warm, double tol, int rule, int maxit,
                    const PcgCont *cont = nullptr, const std::function<void()> &then = nullptr);
bool queue_pcg_f(cfem_ctx *c, float cK, float cM, const float *mcoef, int warm, double tol, int rule, int maxit,
                 const PcgCont *cont, int chunk, const int *halt = nullptr);
PcgResult pcg_result(const Scalars &s);
struct PcgSite {
  Scalars *sc;
  int first_patch, n_patches;
  int64_t first_node, n_nodes;
  float lam, mu;
  double *partials, *partials_up;  // [matvec and init grid][3], [update grid][2]
};
VecParams<float> vec_params(cfem_ctx *c, const PcgSite &S, float *p, float *u);
MvParams<float> site_mv(cfem_ctx *c, const PcgSite &S, float cK, float cM, const float *mcoef);
void launch_init(cfem_ctx *c, const VecParams<float> &P, int warm);
void capture_iterations(cfem_ctx *c, const PcgSite &S, const MvParams<float> &mv, int chunk, unsigned long long cond);
bool add_loop(cfem_ctx *c, cudaGraph_t graph, unsigned initial,
              const std::function<void(cudaGraphConditionalHandle)> &prologue,
              const std::function<void(cudaGraphConditionalHandle)> &capture);
void to_internal_d(cfem_ctx *c, const double *src, double *dst);
void to_caller_d(cfem_ctx *c, const double *src, double *dst);
void to_caller_f(cfem_ctx *c, const float *src, double *dst);
void set_diag_vectors(cfem_ctx *c);
void true_residual(cfem_ctx *c, const double *f, const double *x, double *r, float *r32, double &rr, double &ff);
void true_residual_async(cfem_ctx *c, const double *f, const double *x, double *r, float *r32, double *out2);
void make_rhs(cfem_ctx *c, double a, double b, double *dst);
cfem_status run_guarded(const std::function<cfem_status()> &fn);
void check_ctx(const cfem_ctx *c);
// Calls that take one mesh refuse a context of batched meshes.
inline void single_mesh_only(const cfem_ctx *c) {
  if (c->n_inst)
    throw Fail{CFEM_ERR_UNSUPPORTED, "a context of batched meshes supports cfem_batch_static_solve only"};
}
// Throws if a bulk-copy wait of the edge-fan matvec timed out (synchronises the stream).
// Launch with programmatic stream serialization: the kernel may start while
// the previous kernel in the stream runs (it calls griddep_wait before reading
// that kernel's results). Used for the matvec / update pairs of the PCG loop
// and the kernels of an explicit dynamics step. Every kernel launched this
// way waits for its predecessor before it finishes, so completion stays
// ordered along the stream.
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), dim3 g, dim3 b, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, kern, args...));
}

// The same after the stream has been waited for.
void check_copy_flag(cfem_ctx *c);
void check_copy_error(cfem_ctx *c);
// Whether the kernels may work on a caller's array in place: device memory of
// the context's GPU, aligned to its elements.
bool direct_access(const cfem_ctx *c, const void *p, size_t elem);
// Orders the context's stream after the caller's stream (device inputs written there).
void enter(cfem_ctx *c);
cfem_solve_params default_params();
cfem_status solve_internal(cfem_ctx *c, const cfem_solve_params *prm, cfem_solve_info *info);
void rebuild_operator(cfem_ctx *c);
void build_rows(cfem_ctx *c);
// Slots and counter of a cooperative kernel's exchanges, emptied on the stream.
GridSync start_grid_sync(cfem_ctx *c, int sets);
// y = K' x in FP64 (node vectors, or the caller's arrays; y is overwritten)
void rows_apply(cfem_ctx *c, const double *x, double *y, bool caller_order = false);
void setup_context(cfem_ctx *c, const cfem_mesh *m, const cfem_material *mat, const cfem_options *opt);
void attach_stream(cfem_ctx *c, cudaStream_t s);

template <typename T>
inline MvParams<T> base_mv(cfem_ctx *c) {
  if constexpr (sizeof(T) == 8) return base_mv_d(c); else return base_mv_f(c);
}
template <typename T>
inline PcgResult run_pcg(cfem_ctx *c, Vecs<T> &V, T cK, T cM, const T *mcoef, int warm, double tol, int rule, int maxit) {
  if constexpr (sizeof(T) == 8) return run_pcg_d(c, V, cK, cM, mcoef, warm, tol, rule, maxit);
  else return run_pcg_f(c, cK, cM, mcoef, warm, tol, rule, maxit);
}
template <typename T>
inline void to_internal(cfem_ctx *c, const double *src, T *dst) {
  static_assert(sizeof(T) == 8, "");
  to_internal_d(c, src, dst);
}
template <typename T>
inline void to_caller(cfem_ctx *c, const T *src, double *dst) {
  if constexpr (sizeof(T) == 8) to_caller_d(c, src, dst); else to_caller_f(c, src, dst);
}

}  // namespace detail
}  // namespace cfem
