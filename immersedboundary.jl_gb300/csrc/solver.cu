// libibgb300: handle, setup (Solver), the CNAB advance! step as captured CUDA graphs, and the
// C ABI of include/ibgb300.h and include/ibgb300_ops.h.
//
// Step sequence (reference: src/streamfcn/cnab/timestepping.jl:253-290), FP64:
//   d  trial state   trial_rings -> nonlin_rhs (all levels) -> X(Gamma), X(rhs) -> Y(CN) -> X
//                    -> trial Vort2Flux (curl on level 1 only)
//   e  forces        E(qs1 + q0) -> Binv gemv
//   f  stress        C_D, C_L per body -> device history
//   g  projection    rot(E^T Fb) -> Ainv_1 -> Gamma_1 = Gamma_s1 - (.)   (buffers swap)
//   h  Vort2Flux     coarsify + Poisson solves (all levels at once, or coarse to fine) + curl
// The explicit CN operator A_l, which the reference applies with two sine transforms, is the
// 5-point stencil it diagonalises (I - alpha_l rot curl); it is fused into the nonlinear-term
// kernel, so each level's trial solve is one Poisson-type solve (equal up to round-off).
#include "ib_common.cuh"
#include "mlp.cuh"
#include "ibgb300.h"
#include "ibgb300_learn.h"
#include "ibgb300_ensemble.h"
#include "ibgb300_ops.h"
#include "ibgb300_diag.h"

#include <algorithm>
#include <chrono>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

using namespace ib;

namespace ib {
thread_local Prof* g_prof = nullptr;
thread_local bool g_pdl = false;
}

namespace {

std::mutex g_err_mu;
std::string g_create_err;

constexpr int kQ0Slots = 1024;  // pinned staging slots of per-step base flux

}  // namespace

// steps of every member one ensemble graph launch can carry (ib_ensemble_set_steps_per_launch)
constexpr int kMaxStepsPerLaunch = 8;

struct ib_handle {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t side = nullptr;            // forked branch of a step (curl of finished levels)
  std::vector<cudaEvent_t> fork_ev;       // one per level, plus the join
  Geometry g{};
  double dt = 0, re = 0, beta0 = 1.5, beta1 = -0.5;
  int nbodies = 0, nb = 0, nf = 0;
  int precision = IB_PREC_FP64;
  FxTables axx, axy;               // FP64 passes
  AxisTables<float> axx32, axy32;  // mixed precision: FP32 transform tables
  // state
  double* G[2] = {nullptr, nullptr};
  double* N[2] = {nullptr, nullptr};
  double* psi = nullptr;
  double* q = nullptr;
  double* fb = nullptr;
  double t = 0.0;
  int parity = 0;
  int64_t steps = 0;
  // step scratch
  double *rhs = nullptr, *w1 = nullptr, *w2 = nullptr, *qs1 = nullptr, *qtmp = nullptr, *gtmp = nullptr;
  double *bcn = nullptr, *edges = nullptr, *rings = nullptr;
  // spectral multipliers (column-major in spectral space, x16)
  double *mLap = nullptr, *mCN1 = nullptr, *mCN2 = nullptr;
  float *mLap32 = nullptr, *mCN1_32 = nullptr;  // FP32 copies (mixed precision)
  float *w32 = nullptr, *x032 = nullptr;        // mixed-precision work: transforms and x0
  float *x132 = nullptr;                        // second FP32 part of the iterate (2 sweeps)
  double* r1 = nullptr;                         // first refinement residual (float-float, 2 sweeps)
  double* conv = nullptr;                       // mixed precision: FP64 copy-out buffer of the state
  int refine = 1;                               // refinement sweeps per mixed-precision solve
  int refine_coarse = 2;                        // sweeps of the coarse-level Vort2Flux solves
  int coarse_from = 2;                          // first (0-based) level counted as coarse
  bool wdst = false;                            // both axes use the warp-per-line passes
  bool gdst = false;                            // mixed precision: transforms as tensor-core GEMMs
  bool tuned_levels = false;                    // mixed precision: the order the autotuner chose
  bool fx_solve = false;                        // mixed precision: solves in fixed point
  bool v2f_fx = false;                          // Vort2Flux in fixed point (FP64 handles: always)
  int scheme = IB_SCHEME_CNAB;                  // time stepping (IB_SCHEME_*)
  int rkc_s = 0;                                // Runge-Kutta-Chebyshev: stages and their
  std::vector<double> rkc_mu, rkc_nu, rkc_mut, rkc_gamt;  // coefficients (index = stage)
  double* rkY[2] = {nullptr, nullptr};          // stage values (rotating)
  double* rkF0 = nullptr;                       // F(Y0)
  double *d_alpha_rkc = nullptr, *d_fac_rkc = nullptr;  // per level 1 / (Re hc^2)
  bool cn_pred = false;                         // mixed: trial CN solve refined from Gamma_n,
  double* cprev = nullptr;                      //   the projection from its previous correction
  cudaEvent_t stress_ev[2] = {nullptr, nullptr};  // fork / join of the stress branch
  SineGemm sgx, sgy;                            // their BF16 sine-matrix images (sgemm.cu)
  float* gw32 = nullptr;                        // FP32 work of the GEMM passes
  double *d_one = nullptr, *d_zero = nullptr;   // residual operator coefficients
  // per-level parameters
  double *d_fac = nullptr, *d_q0 = nullptr, *d_inv_hc2 = nullptr, *d_alpha = nullptr;
  double* h_q0 = nullptr;  // pinned [kQ0Slots][2L]
  int q0_slot = 0;
  // bodies
  double *xb = nullptr, *ds = nullptr, *weight = nullptr;
  int *body_start = nullptr, *body_idx = nullptr;
  double *bmat = nullptr, *binv_cm = nullptr, *binv_rm = nullptr, *ftmp = nullptr;
  double *cdcl = nullptr, *stress = nullptr, *hist = nullptr;
  double* h_stress = nullptr;  // host copy of cdcl, then stress, written by the same kernel
  int hist_cap = 4096;
  int* d_counter = nullptr;
  // moving bodies (IB_MOTION_PRESCRIBED)
  int motion = IB_MOTION_STATIC;
  double *xb_body = nullptr, *vb = nullptr, *d_kin = nullptr;
  int* body_of = nullptr;
  double *cg_r = nullptr, *cg_p = nullptr, *cg_Ap = nullptr, *cg_sc = nullptr;
  double *fb_prev = nullptr, *fb_last = nullptr;  // F_{n-2}, F_{n-1} at the start of a step
  double* cg_z = nullptr;                         // preconditioned residual
  learn::Mlp* mlp = nullptr;                      // learned warm start (ib_learn_init)
  // the moving step as captured graphs (one per buffer parity), from the third step on
  bool use_moving_graph = true;
  cudaGraphExec_t mgexec[2] = {nullptr, nullptr};
  uint64_t mg_key = 0;
  cudaStream_t loop_stream = nullptr;             // capture stream of the CG loop body
  double* h_mslot = nullptr;                      // pinned: per step of a launch, base flux [2L] and
                                                  // kinematics [6 nbodies] (kMaxStepsPerLaunch slots)
  double* h_cgout = nullptr;                      // pinned: CG statistics [4] per step of the last launch
  double *d_cgctl = nullptr, *d_cgout = nullptr;
  bool collect = false;                           // record (features, F_n) every moving step
  std::vector<double> cg_res0;                    // initial relative residual of each CG solve
  int precond = IB_PC_NONE;                       // moving-body CG preconditioner
  int pc_refresh = 0;                             // re-assembly period in steps (0: adaptive)
  int pc_base_iters = -1;                         // iterations of the first solve after an assembly
  int64_t pc_step = -1;                           // step of the last assembly
  int pc_assemblies = 0;
  double pc_assembly_s = 0.0;                     // measured duration of the last assembly
  // Schur assembly work buffers, kept between the re-assemblies of a moving handle
  double *asm_G = nullptr, *asm_P = nullptr, *asm_Wa = nullptr, *asm_Wb = nullptr, *asm_Q = nullptr,
         *asm_R = nullptr, *asm_work = nullptr;
  int asm_nc = 0;
  bool asm_fp64 = false;  // assemble a moving handle's preconditioner in FP64 even in mixed mode
  // mixed precision: Vort2Flux with the rings found first and the levels solved in one batch
  bool v2f_levels = false;
  bool v2f_ok = false, v2f_auto = false;  // the grid allows it / the size rule picks it
  RingPlan rplan;
  // setup-time autotuner: modelled step time of each candidate (form * 2 + levels order), ms;
  // -1 where not tried; index (form * 2 + levels) * 2 + (y pass at 8 blocks per SM)
  double tune_ms[12] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1, -1};
  bool tuned = false;
  double pc_excess_iters = 0.0;                   // iterations above the base since then
  double cg_iter_s = 0.0;                         // measured time of one CG iteration (running mean)
  double *Gw = nullptr, *Pw = nullptr, *qw = nullptr, *rings_w = nullptr;
  double* h_sc = nullptr;  // pinned CG scalars read back each iteration
  double cg_tol = 1e-10;
  int cg_maxiter = 5000;
  int warm_start = IB_WARM_PREVIOUS;
  std::vector<int> cg_iters;
  std::vector<double> cg_res;
  // Host memory that kernels write: a call that has waited for its stream reads it without a copy (a copy
  // to pageable memory and its wait took 8 us of a 128^2 step's 270, the three of ib_get_stress 25).
  int* status = nullptr;  // [0] out of grid, [1] non-finite flux, [2] singular Schur matrix, [3] pipeline timeout
  int* d_box = nullptr;   // face box of the body windows (E^T scatter scratch)
  bool box_ready = false; // static bodies: d_box computed once at setup
  cudaGraphExec_t gexec[2] = {nullptr, nullptr};
  bool use_graph = true;
  // programmatic dependent launch inside the static step graph: measured no faster on GB300
  // (1.236 vs 1.227 ms per 1024^2 x 4 mixed step; 1.23 vs 1.14 ms per 512^2 FP64 step), so off
  // unless IBGB300_PDL=1
  bool use_pdl = false;
  int kernels_per_step = 0;
  int64_t device_bytes = 0;
  double setup_ms = 0.0;
  std::string err;
  std::vector<void*> allocs;
  std::mutex op_mu;              // operator calls' work array (OpWork)
  double* op_work = nullptr;
  int64_t op_cap = 0;

  template <typename T>
  cudaError_t alloc(T** p, size_t count) {
    void* v = nullptr;
    cudaError_t e = cudaMalloc(&v, count * sizeof(T) > 0 ? count * sizeof(T) : 16);
    if (e != cudaSuccess) return e;
    device_bytes += (int64_t)(count * sizeof(T));
    allocs.push_back(v);
    *p = (T*)v;
    return cudaMemsetAsync(v, 0, count * sizeof(T) > 0 ? count * sizeof(T) : 16, stream);
  }
};

namespace {

int fail(ib_handle* h, int code, const char* what, cudaError_t e = cudaSuccess) {
  std::string m = what;
  if (e != cudaSuccess) {
    m += ": ";
    m += cudaGetErrorString(e);
  }
  if (h) h->err = m;
  else {
    std::lock_guard<std::mutex> lock(g_err_mu);
    g_create_err = m;
  }
  return code;
}

#define CK(x)                                                        \
  do {                                                               \
    cudaError_t e_ = (x);                                            \
    if (e_ != cudaSuccess) return fail(h, IB_ERR_CUDA, #x, e_);      \
  } while (0)

// cudaError_t-returning variant for the enqueue helpers
#define CE(x)                              \
  do {                                     \
    cudaError_t e_ = (x);                  \
    if (e_ != cudaSuccess) return e_;      \
  } while (0)

// A Poisson-type operator M: the Laplacian (vort2flux) or I + alpha_l L (CN implicit part).
// m64/m32: spectral multipliers (x16, FP64 / FP32) with their per-slot stride; mc, ma: the
// same operator as a stencil, M x = mc x + ma rot(curl(x)), per slot (stride mstep), used by
// the refinement residual of the mixed-precision solve.
struct SolveOp {
  const double* m64;
  const float* m32;
  int64_t mstride;
  const double* mc;
  const double* ma;
  int mstep;
};

SolveOp op_lap(const ib_handle* h) { return {h->mLap, h->mLap32, 0, h->d_zero, h->d_one, 0}; }
SolveOp op_cn_all(const ib_handle* h) { return {h->mCN1, h->mCN1_32, h->g.nG, h->d_one, h->d_alpha, 1}; }
SolveOp op_cn1(const ib_handle* h) { return {h->mCN1, h->mCN1_32, 0, h->d_one, h->d_alpha, 0}; }

// Fixed-point solve of `batch` arrays (double or float-float): out = F2D(m .* F2D(in [+ apply_bc(bc,
// 1)])), optional subtract epilogue out = sub_from - (...).  w: FP64 work of batch arrays (the transposed
// intermediate).  The row-major intermediate is in `out`, or, where that holds sub_from, in h->w2
// (at most nlevels arrays).
template <typename T>
cudaError_t poisson_fx(ib_handle* h, const T* in, T* out, int batch, const T* bc, const SolveOp& op, const T* sub_from,
                       double* w) {
  CE(fx_fwd<T>(h->g, h->axx.d, in, w, batch, bc, h->stream));
  double* t = sub_from == out ? h->w2 : reinterpret_cast<double*>(out);
  if (sub_from == out && batch > h->g.nlev) return cudaErrorInvalidValue;
  CE(fx_ypass(h->g, h->axy.d, w, t, batch, op.m64, op.mstride, 0, h->stream));
  return fx_inv<T>(h->g, h->axx.d, t, out, batch, sub_from, h->stream);
}

// Mixed-precision solve: FP32 sine transforms refined with float-float residuals.
//   x0 = F32 solve(b)
//   sweep 1: r = b - M x0 (df64, fused into the next x pass);  d1 = F32 solve(r)
//   sweep 2 (optional): r = b - M (x0 + d1) with x0 + d1 an exact FP32 pair;  d2 = F32 solve(r)
//   x = x0 + d1 [+ d2] summed in df64 (optionally subtracted from sub_from)
// b, the result and the residual arithmetic are float-float (df64.cuh), so the whole solve runs
// on the FP32 pipe; w32 / x032 / x132: FP32 work of batch arrays.  sweeps = 0 (warp passes
// only) is the transform-only solve x = x0, FP32-accurate, and needs w32 alone.
cudaError_t poisson_mixed(ib_handle* h, const df64* in, df64* out, int batch, const df64* bc, const SolveOp& op,
                          const df64* sub_from, float* w32, float* x032, float* x132, int sweeps,
                          const df64* pred = nullptr, df64* also_sub = nullptr) {
  const Geometry& g = h->g;
  cudaStream_t s = h->stream;
  YPassArgs<float> ya{};
  ya.in1 = w32;
  ya.out = w32;
  ya.batch = batch;
  ya.stride = g.nG;
  ya.m1 = op.m32;
  ya.mstride = op.mstride;
  XArgs a{};
  a.batch = batch;
  a.stride = g.nG;
  a.bcfac = 1.0;
  if (h->gdst) {
    // BF16x3 tensor-core passes (sgemm.cu): the same sweeps as the warp passes below; gw32 holds
    // the prologue rows and the y pass's middle product, w32 the intermediate
    int* st = h->status;
    float* gw = h->gw32;
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProLoad; a.epi = kEpiStore;
    CE(gx_fwd(g, h->sgx, a, gw, st, s));
    CE(gy_pass(g, h->sgy, ya, gw, st, s));
    if (sweeps <= 0) {
      a.in = w32; a.out = out; a.bc = nullptr; a.sub_from = sub_from; a.base = nullptr; a.base2 = nullptr;
      a.epi = sub_from ? kEpiSubAddBase : kEpiAddBase;
      return gx_inv<df64>(g, h->sgx, a, st, s);
    }
    a.in = w32; a.out = x032; a.bc = nullptr;
    CE(gx_inv<float>(g, h->sgx, a, st, s));
    const bool two = sweeps >= 2 && x132;
    df64* r1 = two ? reinterpret_cast<df64*>(h->r1) : nullptr;
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProResid; a.base = x032; a.base2 = nullptr;
    a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep; a.resid_out = r1;
    CE(gx_fwd(g, h->sgx, a, gw, st, s));
    CE(gy_pass(g, h->sgy, ya, gw, st, s));
    a.resid_out = nullptr;
    if (two) {
      a.in = w32; a.out = x132; a.bc = nullptr; a.pro = kProLoad; a.epi = kEpiStore; a.base = nullptr;
      CE(gx_inv<float>(g, h->sgx, a, st, s));
      a.in = r1; a.out = w32; a.bc = nullptr; a.pro = kProResid; a.base = x132; a.base2 = nullptr;
      CE(gx_fwd(g, h->sgx, a, gw, st, s));
      CE(gy_pass(g, h->sgy, ya, gw, st, s));
    }
    a.in = w32; a.out = out; a.bc = nullptr; a.pro = kProLoad; a.sub_from = sub_from;
    a.base = x032; a.base2 = two ? x132 : nullptr;
    a.epi = sub_from ? kEpiSubAddBase : kEpiAddBase;
    return gx_inv<df64>(g, h->sgx, a, st, s);
  }
  if (h->wdst && pred && h->r1 && !sub_from) {
    // from a predictor p (float-float, e.g. the previous step's value of the unknown):
    //   d1 = F32 solve(r0), r0 = b [+ bc] - M p (kept);  d2 = F32 solve(r0 - M d1)
    //   x = p + d1 + d2
    // two transform solves instead of three; the sweeps carry only the change from p
    df64* r1 = reinterpret_cast<df64*>(h->r1);
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProResidD; a.based = pred; a.epi = kEpiStore;
    a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep; a.resid_out = r1;
    CE((wx_fwd<float, df64>(g, h->axx32.d, a, s)));
    CE(wypass<float>(g, h->axy32.d, ya, s));
    XArgs b{};
    b.batch = batch; b.stride = g.nG; b.bcfac = 1.0;
    b.in = w32; b.out = x032; b.pro = kProLoad; b.epi = kEpiStore;
    CE((wx_inv<float, float>(g, h->axx32.d, b, s)));
    b.in = r1; b.out = w32; b.pro = kProResid; b.base = x032; b.mc = op.mc; b.ma = op.ma; b.mstep = op.mstep;
    CE((wx_fwd<float, df64>(g, h->axx32.d, b, s)));
    CE(wypass<float>(g, h->axy32.d, ya, s));
    b = XArgs{};
    b.batch = batch; b.stride = g.nG; b.bcfac = 1.0;
    b.in = w32; b.out = out; b.pro = kProLoad; b.sub_from = pred; b.base = x032; b.epi = kEpiAddTo;
    b.sub2 = also_sub;  // optionally also also_sub -= x, in the same pass
    return wx_inv<float, df64>(g, h->axx32.d, b, s);
  }
  if (h->wdst) {
    // warp-per-line passes; w32 holds the transposed intermediate
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProLoad; a.epi = kEpiStore;
    CE((wx_fwd<float, df64>(g, h->axx32.d, a, s)));
    CE(wypass<float>(g, h->axy32.d, ya, s));
    if (sweeps <= 0) {
      a.in = w32; a.out = out; a.bc = nullptr; a.sub_from = sub_from; a.base = nullptr; a.base2 = nullptr;
      a.epi = sub_from ? kEpiSubAddBase : kEpiAddBase;
      return wx_inv<float, df64>(g, h->axx32.d, a, s);
    }
    a.in = w32; a.out = x032; a.bc = nullptr;
    CE((wx_inv<float, float>(g, h->axx32.d, a, s)));
    const bool two = sweeps >= 2 && x132;
    // sweep 1: r1 = b [+ bc] - M x0, kept in float-float for the second sweep
    df64* r1 = two ? reinterpret_cast<df64*>(h->r1) : nullptr;
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProResid; a.base = x032; a.base2 = nullptr;
    a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep; a.resid_out = r1;
    CE((wx_fwd<float, df64>(g, h->axx32.d, a, s)));
    CE(wypass<float>(g, h->axy32.d, ya, s));
    a.resid_out = nullptr;
    if (two) {
      a.in = w32; a.out = x132; a.bc = nullptr; a.pro = kProLoad; a.epi = kEpiStore; a.base = nullptr;
      CE((wx_inv<float, float>(g, h->axx32.d, a, s)));
      // sweep 2: r2 = b - M (x0 + d1) = r1 - M d1 (the boundary terms are in r1)
      a.in = r1; a.out = w32; a.bc = nullptr; a.pro = kProResid; a.base = x132; a.base2 = nullptr;
      CE((wx_fwd<float, df64>(g, h->axx32.d, a, s)));
      CE(wypass<float>(g, h->axy32.d, ya, s));
    }
    a.in = w32; a.out = out; a.bc = nullptr; a.pro = kProLoad; a.sub_from = sub_from;
    a.base = x032; a.base2 = two ? x132 : nullptr;
    a.epi = sub_from ? kEpiSubAddBase : kEpiAddBase;
    return wx_inv<float, df64>(g, h->axx32.d, a, s);
  }
  // first solve
  a.in = in; a.out = w32; a.bc = bc; a.pro = kProLoad; a.epi = kEpiStore;
  CE((xpass<float, df64, float>(g, h->axx32.d, a, s)));
  CE(ypass<float>(g, h->axy32.d, ya, s));
  a.in = w32; a.out = x032; a.bc = nullptr;
  CE((xpass<float, float, float>(g, h->axx32.d, a, s)));
  const bool two = sweeps >= 2 && x132;
  // sweep 1: residual (df64) fused with the forward transform of the correction
  a.in = in; a.out = w32; a.bc = bc; a.pro = kProResid; a.base = x032; a.base2 = nullptr;
  a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep;
  CE((xpass<float, df64, float>(g, h->axx32.d, a, s)));
  CE(ypass<float>(g, h->axy32.d, ya, s));
  if (two) {
    a.in = w32; a.out = x132; a.bc = nullptr; a.pro = kProLoad; a.epi = kEpiStore; a.base = nullptr;
    CE((xpass<float, float, float>(g, h->axx32.d, a, s)));
    // sweep 2: residual of the FP32 pair x0 + d1
    a.in = in; a.out = w32; a.bc = bc; a.pro = kProResid; a.base = x032; a.base2 = x132;
    CE((xpass<float, df64, float>(g, h->axx32.d, a, s)));
    CE(ypass<float>(g, h->axy32.d, ya, s));
  }
  // x = x0 [+ d1] + correction, in df64 (optionally subtracted from sub_from)
  a.in = w32; a.out = out; a.bc = nullptr; a.pro = kProLoad; a.sub_from = sub_from;
  a.base = x032; a.base2 = two ? x132 : nullptr;
  a.epi = sub_from ? kEpiSubAddBase : kEpiAddBase;
  return xpass<float, float, df64>(g, h->axx32.d, a, s);
}

// Solve with the step's work buffers (batch <= nlevels); the state type picks the precision:
// double -> FP64 transforms, df64 -> the mixed-precision solve.
cudaError_t solve(ib_handle* h, const double* in, double* out, int batch, const double* bc, const SolveOp& op,
                  const double* sub_from) {
  return poisson_fx<double>(h, in, out, batch, bc, op, sub_from, h->w1);
}
cudaError_t solve(ib_handle* h, const df64* in, df64* out, int batch, const df64* bc, const SolveOp& op,
                  const df64* sub_from) {
  if (h->fx_solve) return poisson_fx<df64>(h, in, out, batch, bc, op, sub_from, h->w1);
  return poisson_mixed(h, in, out, batch, bc, op, sub_from, h->w32, h->x032, h->x132, h->refine);
}

// The handle's state arrays hold doubles (FP64 mode) or float-float pairs (mixed mode); both are
// 8 bytes, so one set of allocations serves either and is viewed with the mode's type.
template <typename S>
S* view(double* p) {
  return reinterpret_cast<S*>(p);
}

// Vort2Flux (src/streamfcn/fluid-ops.jl:438-472) on one L-level set.  If q is null only the
// level-1 flux is formed, into q1.  gam is coarsened in place like the reference.
//
// With q given, the curl of each finished level runs on the side stream while the finer levels
// are solved (it reads only that level's psi and ring); the branch joins before returning.
// Mixed-precision Vort2Flux of all levels in one batch (v2f.cu has the ring transfer).  psi and
// rings hold the previous call's results (zero after a state upload without psi), used as
// predictors: the FP32 sweeps then carry only the change since that call.
//   r0 = Gamma + apply_bc(ring_old) - L psi_p (float-float);  d0 = F32 solve(r0)
//   r1 = r0 - L d0; its spectrum; psi_o = psi_p + d0 + S^-1 spec on the quarter lines
//   rings coarse to fine: ring_l = get_bc(psi_o_{l+1}) + harmonic part of the change of
//   ring_{l+1}   (FP64)
//   sweep 1: d1 = F32 inverse of (spec + spectrum of apply_bc(ring - ring_old))
//   sweep 2: r2 = r1 + apply_bc(ring - ring_old) - L d1;  psi = psi_p + d0 + d1 + F32 solve(r2)
// Only level 0 is finished when only its fluxes are asked for (q == nullptr); the other levels
// keep their previous psi.
cudaError_t vort2flux_levels(ib_handle* h, df64* gam, df64* psi, df64* q, df64* q1, df64* rings) {
  const Geometry& g = h->g;
  const int L = g.nlev, ncol = g.nx - 1, nrow = g.ny - 1;
  const int64_t nG = g.nG;
  cudaStream_t s = h->stream;
  const RingPlan& rp = h->rplan;
  const DstAxis<float>& ax = h->axx32.d;
  const DstAxis<float>& ay = h->axy32.d;
  const SolveOp op = op_lap(h);
  const int nf = q ? L : 1;
  df64* r1 = reinterpret_cast<df64*>(h->r1);
  // x and y line transforms side by side (side stream) where there is one.  Only calls that
  // finish every level fork: the level-0-only calls include the Schur products of the CG loop,
  // which may be captured into a graph's conditional body (kernels and copies only).
  const bool fork = q && h->side;
  auto lines2 = [&](const float* inx, int64_t inx_b, float* outx, int64_t outx_b, const float* iny, int64_t iny_b,
                    float* outy, int64_t outy_b, int nl) -> cudaError_t {
    cudaStream_t sy = s;
    if (fork) {
      CE(cudaEventRecord(h->fork_ev[0], s));
      CE(cudaStreamWaitEvent(h->side, h->fork_ev[0], 0));
      sy = h->side;
    }
    CE(v2f_lines(ax, inx, inx_b, ncol, outx, outx_b, ncol, nl, s));
    CE(v2f_lines(ay, iny, iny_b, nrow, outy, outy_b, nrow, nl, sy));
    if (fork) {
      CE(cudaEventRecord(h->fork_ev[1], h->side));
      CE(cudaStreamWaitEvent(s, h->fork_ev[1], 0));
    }
    return cudaSuccess;
  };
  for (int l = 1; l < L; ++l) CE(coarsify<df64>(g, gam + l * nG, gam + (l - 1) * nG, 1, nG, s));
  XArgs a{};
  a.batch = L; a.stride = nG; a.bcfac = 1.0;
  a.in = gam; a.out = h->w32; a.bc = rings; a.pro = kProResidD; a.based = psi; a.epi = kEpiStore;
  a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep; a.resid_out = r1;
  CE((wx_fwd<float, df64>(g, ax, a, s)));
  YPassArgs<float> ya{};
  ya.in1 = h->w32; ya.out = h->w32; ya.batch = L; ya.stride = nG; ya.m1 = op.m32; ya.mstride = op.mstride;
  CE(wypass<float>(g, ay, ya, s));
  a = XArgs{};
  a.batch = L; a.stride = nG; a.bcfac = 1.0;
  a.in = h->w32; a.out = h->x032; a.pro = kProLoad; a.epi = kEpiStore;
  CE((wx_inv<float, float>(g, ax, a, s)));
  a.in = r1; a.out = h->w32; a.pro = kProResid; a.base = h->x032; a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep;
  a.resid_out = r1;
  CE((wx_fwd<float, df64>(g, ax, a, s)));
  CE(v2f_yspec(g, ay, h->w32, op.m32, L, rp.vrow, s));
  CE(v2f_colsum(g, rp, h->w32, L, s));
  CE(lines2(rp.vrow, 2 * ncol, rp.qline, rp.qls, rp.ucol, 2 * nrow, rp.qline + 2 * ncol, rp.qls, 2 * L));
  for (int l = L - 2; l >= 0; --l) {
    CE(v2f_ring_eval(g, rp, l, psi + (l + 1) * nG, h->x032 + (l + 1) * nG, rings + (int64_t)l * g.nbc, s));
    if (l > 0) CE(v2f_ring_coef(g, rp, l, s));
  }
  const int ns = std::min(nf, L - 1);  // finished levels with a ring
  CE(lines2(rp.sidex, 2 * ncol, rp.sidex, 2 * ncol, rp.sidey, 2 * nrow, rp.sidey, 2 * nrow, 2 * ns));
  CE(v2f_yring(g, ay, ax, h->w32, op.m32, nf, rp.sidex, rp.sidey, s));
  a = XArgs{};
  a.batch = nf; a.stride = nG; a.bcfac = 1.0;
  a.in = h->w32; a.out = h->x132; a.pro = kProLoad; a.epi = kEpiStore;
  CE((wx_inv<float, float>(g, ax, a, s)));
  if (ns > 0) CE(apply_bc<df64>(g, r1, reinterpret_cast<const df64*>(rp.dring), df64(1.0f), ns, s));
  a.in = r1; a.out = h->w32; a.pro = kProResid; a.base = h->x132; a.mc = op.mc; a.ma = op.ma; a.mstep = op.mstep;
  CE((wx_fwd<float, df64>(g, ax, a, s)));
  ya.batch = nf;
  CE(wypass<float>(g, ay, ya, s));
  a = XArgs{};
  a.batch = nf; a.stride = nG; a.bcfac = 1.0;
  a.in = h->w32; a.out = psi; a.sub_from = psi; a.pro = kProLoad; a.base = h->x032; a.base2 = h->x132;
  a.epi = kEpiAddTo;
  CE((wx_inv<float, df64>(g, ax, a, s)));
  return q ? curl<df64>(g, psi, rings, q, L, s) : curl<df64>(g, psi, rings, q1, 1, s);
}

// Vort2Flux of all levels in one batch, in fixed point: no predictor and no sweeps, the rings as in
// vort2flux_levels.
//   spectra of Gamma / L of every level with zero rings (in w1), their sums for the quarter lines, the
//   lines; rings coarse to fine; the rings' own spectrum added on the way back
// The spectra stay in FP64, so the lines and rings carry no more error than a solve (2e-15 of psi apart
// from the other order at 256^2, 8e-15 at 1024^2).  Against the level-by-level order it runs one chain of passes where that runs one per level, and a
// call that wants the finest level's fluxes alone (the trial state, B's products) leaves out half of
// the coarser levels' passes.
template <typename S>
cudaError_t vort2flux_fx(ib_handle* h, S* gam, S* psi, S* q, S* q1, S* rings, bool may_fork) {
  const Geometry& g = h->g;
  const int L = g.nlev, ncol = g.nx - 1;
  const int64_t nG = g.nG;
  cudaStream_t s = h->stream;
  const RingPlan& rp = h->rplan;
  const int nf = q ? L : 1;               // finished levels
  const int ns = std::min(nf, L - 1);     // of them, those with a ring
  const bool fork = may_fork && h->side;
  // transforms of m levels' quarter lines or ring sides (2 along x, 2 along y each), in place: as the
  // rows of one array on a square grid; else of two, side by side where there is a side stream
  auto lines = [&](double* v, int m) -> cudaError_t {
    Geometry gx = g, gy = g;
    gx.nG = gy.nG = rp.qls;
    gx.ny = gy.ny = 3;
    gy.nx = g.ny;
    if (g.nx == g.ny) {
      gx.ny = 5;
      return fx_inv<double>(gx, h->axx.d, v, v, m, nullptr, s);
    }
    cudaStream_t sy = s;
    if (fork) {
      CE(cudaEventRecord(h->fork_ev[0], s));
      CE(cudaStreamWaitEvent(h->side, h->fork_ev[0], 0));
      sy = h->side;
    }
    CE(fx_inv<double>(gx, h->axx.d, v, v, m, nullptr, s));
    CE(fx_inv<double>(gy, h->axy.d, v + 2 * ncol, v + 2 * ncol, m, nullptr, sy));
    if (fork) {
      CE(cudaEventRecord(h->fork_ev[1], h->side));
      CE(cudaStreamWaitEvent(s, h->fork_ev[1], 0));
    }
    return cudaSuccess;
  };
  for (int l = 1; l < L; ++l) CE(coarsify<S>(g, gam + l * nG, gam + (l - 1) * nG, 1, nG, s));
  CE(fx_fwd<S>(g, h->axx.d, gam, h->w1, L, nullptr, s));
  CE(fx_yspec(g, h->axy.d, h->w1, L, h->mLap, rp.qfx, rp.qls, s));
  CE(v2f_fx_colsum(g, rp, h->w1, s));
  CE(lines(rp.qfx, L - 1));
  CE(v2f_fx_rings<S>(g, rp, rings, s));
  CE(lines(rp.side, ns));
  const FxRings r{ns, rp.side, rp.sinx, rp.siny};
  double* t = reinterpret_cast<double*>(psi);
  CE(fx_yring(g, h->axy.d, h->w1, t, nf, h->mLap, r, s));
  CE(fx_inv<S>(g, h->axx.d, t, psi, nf, nullptr, s));
  return q ? curl<S>(g, psi, rings, q, L, s) : curl<S>(g, psi, rings, q1, 1, s);
}

// may_fork: whether the side stream may be used (not where a conditional graph body is captured)
template <typename S>
cudaError_t vort2flux(ib_handle* h, S* gam, S* psi, S* q, S* q1, S* rings, bool may_fork = true) {
  if (h->v2f_levels && h->v2f_fx) return vort2flux_fx(h, gam, psi, q, q1, rings, may_fork);
  if constexpr (std::is_same<S, df64>::value) {
    if (h->v2f_levels) return vort2flux_levels(h, gam, psi, q, q1, rings);
  }
  // one level's solve: FP64 and fixed-point handles alike, or the FP32 passes
  auto level_solve = [&](const S* in, S* out, const S* ring, int sweeps) -> cudaError_t {
    if constexpr (std::is_same<S, df64>::value) {
      if (!h->v2f_fx)
        return poisson_mixed(h, in, out, 1, ring, op_lap(h), nullptr, h->w32, h->x032, h->x132,
                             sweeps > 0 ? sweeps : h->refine);
    }
    return poisson_fx<S>(h, in, out, 1, ring, op_lap(h), nullptr, h->w1);
  };
  const Geometry& g = h->g;
  const int L = g.nlev;
  const int64_t nG = g.nG;
  cudaStream_t s = h->stream;
  const bool fork = q && h->side && L > 1;
  auto curl_level = [&](int l, const S* ring) -> cudaError_t {
    if (!fork) return curl<S>(g, psi + l * nG, ring, q + (int64_t)l * g.nq, 1, s);
    CE(cudaEventRecord(h->fork_ev[l], s));
    CE(cudaStreamWaitEvent(h->side, h->fork_ev[l], 0));
    return curl<S>(g, psi + l * nG, ring, q + (int64_t)l * g.nq, 1, h->side);
  };
  for (int l = 1; l < L; ++l) CE(coarsify<S>(g, gam + l * nG, gam + (l - 1) * nG, 1, nG, s));
  // mixed precision: the coarse levels only feed the finer levels' boundary rings
  const int coarse = std::min(h->refine, h->refine_coarse);
  CE(level_solve(gam + (L - 1) * nG, psi + (L - 1) * nG, nullptr, L - 1 >= h->coarse_from ? coarse : 0));
  if (q) CE(curl_level(L - 1, nullptr));
  else if (L == 1) CE(curl<S>(g, psi, nullptr, q1, 1, s));
  for (int l = L - 2; l >= 0; --l) {
    S* ring = rings + (int64_t)l * g.nbc;
    CE(get_bc<S>(g, psi + (l + 1) * nG, ring, 1, S(1.0), s));
    CE(level_solve(gam + l * nG, psi + l * nG, ring, l >= h->coarse_from ? coarse : 0));
    if (q) CE(l > 0 ? curl_level(l, ring) : curl<S>(g, psi, ring, q, 1, s));
    else if (l == 0) CE(curl<S>(g, psi, ring, q1, 1, s));
  }
  if (fork) {
    CE(cudaEventRecord(h->fork_ev[L], h->side));
    CE(cudaStreamWaitEvent(s, h->fork_ev[L], 0));
  }
  return cudaSuccess;
}

__global__ void k_hist_append(const double* __restrict__ cdcl, double* __restrict__ hist, int cap, int n,
                              int* __restrict__ counter) {
  pdl_begin();
  const int idx = *counter % cap;
  for (int i = threadIdx.x; i < n; i += blockDim.x) hist[(int64_t)idx * n + i] = cdcl[i];
  __syncthreads();
  if (threadIdx.x == 0) *counter = *counter + 1;
}

// state conversions of the mixed mode: in place double -> df64, and df64 -> double
__global__ void k_to_df64(double* p, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const double v = p[t];
    reinterpret_cast<df64*>(p)[t] = df64(v);
  }
}
__global__ void k_from_df64(const df64* __restrict__ in, double* __restrict__ out, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = static_cast<double>(in[t]);
}
int conv_blocks(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return (int)(b > 4096 ? 4096 : (b < 1 ? 1 : b));
}

// Enqueue one advance! for buffer parity p (see the file header).
// d. trial state (GetTrialState, timestepping.jl:28-79): Gamma_s into the other Gamma buffer,
// psi on every level and the trial flux on level 1 (the only level the step reads)
template <typename S>
cudaError_t enqueue_trial(ib_handle* h, int p) {
  ib::Range nvtx_range("trial state");
  const Geometry& g = h->g;
  const int L = g.nlev;
  cudaStream_t s = h->stream;
  S* gam = view<S>(h->G[p]);
  S* gs = view<S>(h->G[p ^ 1]);
  CE(trial_rings<S>(g, gam, view<S>(h->bcn), view<S>(h->edges), h->d_fac, s));
  NonlinArgs<S> na{};
  na.q = view<S>(h->q);
  na.gamma = gam;
  na.bcn = view<S>(h->bcn);
  na.nl_old = view<S>(h->N[p ^ 1]);
  na.edges = view<S>(h->edges);
  na.nl_new = view<S>(h->N[p]);
  na.rhs = view<S>(h->rhs);
  na.q0 = h->d_q0;
  na.inv_hc2 = h->d_inv_hc2;
  na.alpha = h->d_alpha;
  na.dtb0 = h->dt * h->beta0;
  na.dtb1 = h->dt * h->beta1;
  CE(nonlin_rhs<S>(g, na, s));
  // Gamma_s[l] = Ainv_l rhs[l] for every level in one batched solve (mixed precision: refined
  // from Gamma_n[l], the change over one step being what the FP32 sweeps carry)
  if constexpr (std::is_same<S, df64>::value) {
    if (h->cn_pred && !h->fx_solve)
      CE(poisson_mixed(h, view<S>(h->rhs), gs, L, nullptr, op_cn_all(h), nullptr, h->w32, h->x032, h->x132, 2, gam));
    else
      CE(solve(h, view<S>(h->rhs), gs, L, nullptr, op_cn_all(h), nullptr));
  } else {
    CE(solve(h, view<S>(h->rhs), gs, L, nullptr, op_cn_all(h), nullptr));
  }
  return vort2flux<S>(h, gs, view<S>(h->psi), nullptr, view<S>(h->qs1), view<S>(h->rings));
}

// f. update_stress! (states.jl:53-84) and the device C_D / C_L history
cudaError_t enqueue_stress(ib_handle* h) {
  ib::Range nvtx_range("stress");
  cudaStream_t s = h->stream;
  CE(update_stress_hd(h->fb, h->nb, h->nbodies, h->body_start, h->ds, h->g.h, h->dt, h->cdcl, h->stress,
                      h->h_stress, s));
  return launch_k(k_hist_append, dim3(1), dim3(64), 0, s, (const double*)h->cdcl, h->hist, h->hist_cap, 2 * h->nbodies,
                  h->d_counter);
}

// g. CircProjecter (timestepping.jl:156-171): Gamma_1 = Gamma_s1 - Ainv_1 C^T E^T Fb, then
// h. Vort2Flux on the new state (timestepping.jl:285); the trial buffer becomes Gamma
template <typename S>
cudaError_t enqueue_project(ib_handle* h, int p) {
  ib::Range nvtx_range("projection");
  const Geometry& g = h->g;
  S* gs = view<S>(h->G[p ^ 1]);
  if (h->nb > 0) {
    CE(reg_scatter_rot<S>(g, h->fb, h->body_idx, h->weight, h->nb, view<S>(h->qtmp), view<S>(h->gtmp), 1, h->nf,
                          h->status + 1, h->d_box, h->box_ready, h->stream));
    bool done = false;
    if constexpr (std::is_same<S, df64>::value) {
      if (h->cprev && h->wdst && h->r1) {
        // c = Ainv_1 C^T E^T Fb refined from the previous step's c (kept in cprev), then
        // Gamma_s1 -= c
        df64* c = view<df64>(h->cprev);
        CE(poisson_mixed(h, view<S>(h->gtmp), c, 1, nullptr, op_cn1(h), nullptr, h->w32, h->x032, h->x132, 2, c, gs));
        done = true;
      }
    }
    if (!done) CE(solve(h, view<S>(h->gtmp), gs, 1, nullptr, op_cn1(h), gs));
  }
  return vort2flux<S>(h, gs, view<S>(h->psi), view<S>(h->q), nullptr, view<S>(h->rings));
}

// Enqueue one advance! for bodies fixed in the grid (buffer parity p, see the file header).
template <typename S>
cudaError_t enqueue_step(ib_handle* h, int p) {
  CE(enqueue_trial<S>(h, p));
  if (h->nb > 0) {
    // e. BoundaryForcer{RigidBody{GridFrame}} (timestepping.jl:106-120)
    CE(reg_gather<S>(h->g, view<S>(h->qs1), h->d_q0, h->body_idx, h->weight, h->nb, h->ftmp, 1, h->g.nq, h->nf,
                     h->stream));
    CE(gemv_rowmajor(h->binv_rm, h->ftmp, h->fb, h->nf, h->stream));
    if (h->side && h->stress_ev[0]) {
      // C_D / C_L and the surface stress only read Fb: a branch beside the projection
      CE(cudaEventRecord(h->stress_ev[0], h->stream));
      CE(cudaStreamWaitEvent(h->side, h->stress_ev[0], 0));
      cudaStream_t main = h->stream;
      h->stream = h->side;
      const cudaError_t es = enqueue_stress(h);
      h->stream = main;
      CE(es);
      CE(cudaEventRecord(h->stress_ev[1], h->side));
      CE(enqueue_project<S>(h, p));
      return cudaStreamWaitEvent(h->stream, h->stress_ev[1], 0);
    }
    CE(enqueue_stress(h));
  }
  return enqueue_project<S>(h, p);
}

// One step of the Runge-Kutta-Chebyshev scheme (FP64, bodies fixed in the grid), buffer parity p:
//   Y0 = Gamma_n;  Y1 = Y0 + mut_1 dt F(Y0);
//   Y_j = (1 - mu_j - nu_j) Y0 + mu_j Y_{j-1} + nu_j Y_{j-2} + mut_j dt F(Y_{j-1}) + gamt_j dt F(Y0)
//   F(Y) = N(Y) + (1/(Re hc^2)) (ring edges - lap5 Y) per level: the CNAB scheme's nonlinear
//   term (with its rings) and the explicit viscous term, whose missing neighbours at a level's
//   edges are the next coarser level's values (get_bc!); N and the fluxes of Y_{j-1} from a
//   Vort2Flux of every level (which coarsifies Y_{j-1} in place, as the reference's does to Gamma)
//   Fb = B'^-1 E(q(Y_s) + q0), B' = E C Lap^-1 C^T E^T;  Gamma_{n+1} = Y_s - C^T E^T Fb on level 1
cudaError_t enqueue_rkc_step(ib_handle* h, int p) {
  ib::Range nvtx_range("RKC step");
  const Geometry& g = h->g;
  const int L = g.nlev;
  const int64_t n = (int64_t)L * g.nG;
  cudaStream_t s = h->stream;
  double* Y0 = h->G[p];
  double* out = h->G[p ^ 1];
  const double dt = h->dt;
  // rhs = Y + F(Y), from the fluxes q of Y
  auto evalG = [&](const double* Y, const double* q) -> cudaError_t {
    CE(trial_rings<double>(g, Y, h->bcn, h->edges, h->d_fac_rkc, s, false));
    NonlinArgs<double> na{};
    na.q = q;
    na.gamma = Y;
    na.bcn = h->bcn;
    na.nl_old = h->N[p];      // weight 0
    na.edges = h->edges;
    na.nl_new = h->N[p ^ 1];  // N(Y) (not kept: the scheme has no history)
    na.rhs = h->rhs;
    na.q0 = h->d_q0;
    na.inv_hc2 = h->d_inv_hc2;
    na.alpha = h->d_alpha_rkc;
    na.dtb0 = 1.0;
    na.dtb1 = 0.0;
    return nonlin_rhs<double>(g, na, s);
  };
  const int S = h->rkc_s;
  CE(evalG(Y0, h->q));
  double* first = S == 1 ? out : h->rkY[0];
  CE(rkc_stage(n, first, Y0, Y0, nullptr, h->rhs, h->rkF0, 1.0, 0.0, 0.0, h->rkc_mut[1] * dt, 0.0, true, s));
  double *Ym1 = first, *Ym2 = Y0;
  for (int j = 2; j <= S; ++j) {
    CE(vort2flux<double>(h, Ym1, h->psi, h->q, nullptr, h->rings));
    CE(evalG(Ym1, h->q));
    double* dst = (j == S) ? out : (j == 2 ? h->rkY[1] : Ym2);
    const double mu = h->rkc_mu[j], nu = h->rkc_nu[j];
    CE(rkc_stage(n, dst, Y0, Ym1, Ym2, h->rhs, h->rkF0, 1.0 - mu - nu, mu, nu, h->rkc_mut[j] * dt,
                 h->rkc_gamt[j] * dt, false, s));
    Ym2 = Ym1;
    Ym1 = dst;
  }
  if (h->nb > 0) {
    CE(vort2flux<double>(h, out, h->psi, nullptr, h->qs1, h->rings));
    CE(reg_gather<double>(g, h->qs1, h->d_q0, h->body_idx, h->weight, h->nb, h->ftmp, 1, g.nq, h->nf, s));
    CE(gemv_rowmajor(h->binv_rm, h->ftmp, h->fb, h->nf, s));
    CE(enqueue_stress(h));
    CE(reg_scatter_rot<double>(g, h->fb, h->body_idx, h->weight, h->nb, h->qtmp, h->gtmp, 1, h->nf, h->status + 1,
                               h->d_box, h->box_ready, s));
    CE(axpby<double>(out, h->gtmp, -1.0, 1.0, g.nG, s));
  }
  return vort2flux<double>(h, out, h->psi, h->q, nullptr, h->rings);
}

cudaError_t enqueue_step_mode(ib_handle* h, int p) {
  if (h->scheme == IB_SCHEME_RKC) return enqueue_rkc_step(h, p);
  return h->precision == IB_PREC_MIXED ? enqueue_step<df64>(h, p) : enqueue_step<double>(h, p);
}

// Second-order Runge-Kutta-Chebyshev coefficients with damping eps = 2/13 (Sommeijer, Shampine
// and Verwer, "RKC: an explicit solver for parabolic PDEs", 1998), from the Chebyshev
// polynomials T_j and their derivatives at w0 = 1 + eps / s^2.  Returns the length beta(s) of
// the stability interval on the negative real axis.
double rkc_coefficients(int S, std::vector<double>& mu, std::vector<double>& nu, std::vector<double>& mut,
                        std::vector<double>& gamt) {
  const double eps = 2.0 / 13.0, w0 = 1.0 + eps / ((double)S * S);
  std::vector<double> T(S + 1), T1(S + 1), T2(S + 1);
  T[0] = 1.0; T[1] = w0;
  T1[0] = 0.0; T1[1] = 1.0;
  T2[0] = 0.0; T2[1] = 0.0;
  for (int j = 2; j <= S; ++j) {
    T[j] = 2.0 * w0 * T[j - 1] - T[j - 2];
    T1[j] = 2.0 * T[j - 1] + 2.0 * w0 * T1[j - 1] - T1[j - 2];
    T2[j] = 4.0 * T1[j - 1] + 2.0 * w0 * T2[j - 1] - T2[j - 2];
  }
  const double w1 = T1[S] / T2[S];
  std::vector<double> b(S + 1);
  for (int j = 2; j <= S; ++j) b[j] = T2[j] / (T1[j] * T1[j]);
  b[0] = b[1] = b[2];
  mu.assign(S + 1, 0.0); nu.assign(S + 1, 0.0); mut.assign(S + 1, 0.0); gamt.assign(S + 1, 0.0);
  mut[1] = b[1] * w1;
  for (int j = 2; j <= S; ++j) {
    mu[j] = 2.0 * b[j] * w0 / b[j - 1];
    nu[j] = -b[j] / b[j - 2];
    mut[j] = 2.0 * b[j] * w1 / b[j - 1];
    gamt[j] = -(1.0 - b[j - 1] * T[j - 1]) * mut[j];
  }
  return (w0 + 1.0) * T2[S] / T1[S];
}

// B z for the current weights (B_Times, cnab/ops.jl:125-143): E q1(Vort2Flux(Ainv_1 C^T E^T z)).
template <typename S>
cudaError_t schur_apply(ib_handle* h, const double* z, double* out) {
  const Geometry& g = h->g;
  cudaStream_t s = h->stream;
  S* Gw = view<S>(h->Gw);
  CE(reg_scatter_rot<S>(g, z, h->body_idx, h->weight, h->nb, view<S>(h->qtmp), view<S>(h->gtmp), 1, h->nf,
                        h->status + 1, h->d_box, h->box_ready, s));
  CE(solve(h, view<S>(h->gtmp), Gw, 1, nullptr, op_cn1(h), nullptr));
  if (g.nlev > 1) CE(cudaMemsetAsync(Gw + g.nG, 0, sizeof(S) * (g.nlev - 1) * g.nG, s));
  CE(vort2flux<S>(h, Gw, view<S>(h->Pw), nullptr, view<S>(h->qw), view<S>(h->rings_w), false));
  return reg_gather<S>(g, view<S>(h->qw), nullptr, h->body_idx, h->weight, h->nb, out, 1, g.nq, h->nf, s);
}

int check_status(ib_handle* h) {
  CK(cudaStreamSynchronize(h->stream));
  const volatile int* st = h->status;
  if (st[0]) return fail(h, IB_ERR_BODY_OUT_OF_GRID, "body point within 7 cells of the finest-grid edge");
  if (st[1]) return fail(h, IB_ERR_NONFINITE, "infinite flux");
  if (st[2]) return fail(h, IB_ERR_SINGULAR, "zero or non-finite pivot in the Schur matrix");
  if (st[3]) return fail(h, IB_ERR_TIMEOUT, "a tensor-core kernel gave up waiting for its pipeline");
  return IB_OK;
}

// host copy of the spectral multipliers, x16 for the F-convention transforms
void build_multipliers(const ib_handle* h, std::vector<double>& lap, std::vector<double>& cn1,
                       std::vector<double>& cn2) {
  const Geometry& g = h->g;
  const int nx = g.nx, ny = g.ny, ncol = nx - 1, nrow = ny - 1;
  const double pi = 3.14159265358979323846;
  const double scale = 1.0 / (4.0 * nx * ny);
  std::vector<double> ci(ncol), cj(nrow);
  for (int i = 0; i < ncol; ++i) ci[i] = std::cos(pi * (double)(i + 1) / nx);
  for (int j = 0; j < nrow; ++j) cj[j] = std::cos(pi * (double)(j + 1) / ny);
  lap.assign((size_t)ncol * nrow, 0.0);
  cn1.assign((size_t)g.nlev * ncol * nrow, 0.0);
  cn2.assign((size_t)g.nlev * ncol * nrow, 0.0);
  for (int I = 0; I < ncol; ++I)
    for (int J = 0; J < nrow; ++J) {
      const double lam = -2.0 * (ci[I] + cj[J] - 2.0);  // lap_eigs, fluid-ops.jl:58-61
      const size_t idx = (size_t)I * nrow + J;           // spectral column-major
      lap[idx] = 16.0 * (scale / lam);
      for (int l = 0; l < g.nlev; ++l) {
        const double hc = g.h * std::ldexp(1.0, l);
        const double expl = 1.0 / (1.0 - lam * h->dt / (2.0 * h->re * (hc * hc)));  // cnab/ops.jl:26
        const double impl = 1.0 + lam * h->dt / (2.0 * h->re * (hc * hc));          // cnab/ops.jl:29
        cn1[(size_t)l * ncol * nrow + idx] = 16.0 * (scale / impl);
        cn2[(size_t)l * ncol * nrow + idx] = 1.0 / expl;
      }
    }
}

// Columns c0 .. c0+n-1 of B (B_Times, cnab/ops.jl:125-143 on unit vectors) into h->bmat.  S =
// double: FP64 solves; S = df64: transform-only FP32 solves (sweeps 0 on the warp passes, one
// sweep otherwise), B to FP32 accuracy.  Buffers hold n arrays per level (Gb, Pb: L n), Wb is
// the solves' work (n FP64 arrays, or 2n FP32 ones).
template <typename S>
cudaError_t schur_columns(ib_handle* h, int c0, int n, double* Wa, double* Gb, double* Pb, double* Wb, double* Qb,
                          double* Rb) {
  const Geometry& g = h->g;
  const int L = g.nlev, nf = h->nf;
  const int64_t nG = g.nG;
  cudaStream_t s = h->stream;
  auto psolve = [&](const S* in, S* out, const S* bc, const SolveOp& op) -> cudaError_t {
    if constexpr (std::is_same<S, double>::value) {
      return poisson_fx<double>(h, in, out, n, bc, op, nullptr, Wb);
    } else {
      float* w = reinterpret_cast<float*>(Wb);
      return poisson_mixed(h, in, out, n, bc, op, nullptr, w, w + (int64_t)n * nG, nullptr, h->wdst ? 0 : 1);
    }
  };
  S *A = view<S>(Wa), *G = view<S>(Gb), *P = view<S>(Pb), *Q = view<S>(Qb), *R = view<S>(Rb);
  CE(unit_scatter_rot<S>(g, h->body_idx, h->weight, h->nb, c0, n, A, s));
  if (h->scheme == IB_SCHEME_RKC)  // explicit scheme: B' = E C Lap^-1 C^T E^T, no implicit operator
    CE(cudaMemcpyAsync(G, A, sizeof(S) * n * nG, cudaMemcpyDeviceToDevice, s));
  else
    CE(psolve(A, G, nullptr, op_cn1(h)));
  if (L > 1) CE(cudaMemsetAsync(G + (int64_t)n * nG, 0, sizeof(S) * (L - 1) * n * nG, s));
  for (int l = 1; l < L; ++l) CE(coarsify<S>(g, G + (int64_t)l * n * nG, G + (int64_t)(l - 1) * n * nG, n, nG, s));
  CE(psolve(G + (int64_t)(L - 1) * n * nG, P + (int64_t)(L - 1) * n * nG, nullptr, op_lap(h)));
  for (int l = L - 2; l >= 0; --l) {
    CE(get_bc<S>(g, P + (int64_t)(l + 1) * n * nG, R, n, S(1.0), s));
    CE(psolve(G + (int64_t)l * n * nG, P + (int64_t)l * n * nG, R, op_lap(h)));
  }
  CE(curl<S>(g, P, L > 1 ? R : nullptr, Q, n, s));
  return reg_gather<S>(g, Q, nullptr, h->body_idx, h->weight, h->nb, h->bmat + (int64_t)c0 * nf, n, g.nq, nf, s);
}

// Schur matrix assembly (cnab/ops.jl:79-94 with B_Times, ops.jl:125-143), `nc` columns per
// batch of device solves; then inverse (ops.jl:96) and a row-major copy for the step's gemv.
// The B of bodies fixed in the grid is the direct solve and is assembled in FP64; for moving
// bodies B^-1 only preconditions CG on the exact operator, and a mixed-precision handle
// assembles it with FP32 transforms.
int assemble_schur(ib_handle* h) {
  ib::Range nvtx_range("assemble Schur inverse");
  const Geometry& g = h->g;
  const int L = g.nlev, nf = h->nf;
  const int64_t nG = g.nG;
  size_t freeb = 0, totb = 0;
  CK(cudaMemGetInfo(&freeb, &totb));
  const double per_col = 8.0 * ((2.0 * L + 2.0) * nG + g.nq + g.nbc);
  double budget = 0.25 * (double)freeb;
  if (budget > 16e9) budget = 16e9;
  int nc = (int)(budget / per_col);
  if (nc > 64) nc = 64;
  if (nc > nf) nc = nf;
  if (nc < 1) return fail(h, IB_ERR_CUDA, "not enough device memory for the Schur assembly");
  // a moving handle keeps its buffers for the next re-assembly; a static one frees them
  const bool keep = h->motion == IB_MOTION_PRESCRIBED;
  if (keep && h->asm_G) nc = h->asm_nc;
  double *Gb = h->asm_G, *Pb = h->asm_P, *Wa = h->asm_Wa, *Wb = h->asm_Wb, *Qb = h->asm_Q, *Rb = h->asm_R;
  double* work = h->asm_work;
  if (!(keep && h->asm_G)) {
    CK(cudaMalloc(&Gb, sizeof(double) * L * nc * nG));
    CK(cudaMalloc(&Pb, sizeof(double) * L * nc * nG));
    CK(cudaMalloc(&Wa, sizeof(double) * nc * nG));
    CK(cudaMalloc(&Wb, sizeof(double) * nc * nG));
    CK(cudaMalloc(&Qb, sizeof(double) * nc * g.nq));
    CK(cudaMalloc(&Rb, sizeof(double) * nc * g.nbc));
    CK(cudaMalloc(&work, invert_workspace_bytes(nf)));
    if (keep) {
      h->asm_G = Gb; h->asm_P = Pb; h->asm_Wa = Wa; h->asm_Wb = Wb; h->asm_Q = Qb; h->asm_R = Rb;
      h->asm_work = work;
      h->asm_nc = nc;
    }
  }
  auto release = [&]() {
    if (keep) return;
    cudaFree(Gb); cudaFree(Pb); cudaFree(Wa); cudaFree(Wb); cudaFree(Qb); cudaFree(Rb); cudaFree(work);
  };
  cudaStream_t s = h->stream;
  const bool fp32 = keep && h->precision == IB_PREC_MIXED && !h->asm_fp64;
  int rc = IB_OK;
  for (int c0 = 0; c0 < nf && rc == IB_OK; c0 += nc) {
    const int n = (nf - c0 < nc) ? nf - c0 : nc;
    cudaError_t e = fp32 ? schur_columns<df64>(h, c0, n, Wa, Gb, Pb, Wb, Qb, Rb)
                         : schur_columns<double>(h, c0, n, Wa, Gb, Pb, Wb, Qb, Rb);
    if (e != cudaSuccess) rc = fail(h, IB_ERR_CUDA, "Schur assembly", e);
  }
  if (rc != IB_OK) {
    cudaStreamSynchronize(s);
    release();
    return rc;
  }
  // inverse (column-major), then the row-major copy
  cudaError_t e = cudaMemcpyAsync(h->binv_cm, h->bmat, sizeof(double) * (size_t)nf * nf, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = invert_inplace(h->binv_cm, nf, work, h->status + 2, s);
  // column-major (nf x nf) read as row-major is the transpose: transpose it back
  if (e == cudaSuccess) e = transpose(h->binv_cm, h->binv_rm, nf, nf, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  release();
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "Schur inverse", e);
  if (e2 != cudaSuccess) return fail(h, IB_ERR_CUDA, "Schur assembly", e2);
  return IB_OK;
}

// Launch every kernel variant once outside of any capture (sets shared-memory attributes).
int prime_kernels(ib_handle* h) {
  const Geometry& g = h->g;
  CK(poisson_fx<double>(h, h->w2, h->w2, 1, h->rings, op_lap(h), nullptr, h->w1));
  CK(poisson_fx<double>(h, h->w2, h->w2, 1, nullptr, op_lap(h), h->w2, h->w1));
  CK(fx_yspec(g, h->axy.d, h->w1, 1, h->mLap, h->w2, 0, h->stream));
  CK(fx_yring(g, h->axy.d, h->w1, h->w2, 1, h->mLap, FxRings{}, h->stream));
  {  // x and y lines of the all-levels Vort2Flux (a row pass along y too)
    Geometry gy = g;
    gy.nx = g.ny;
    gy.ny = 2;
    CK(fx_inv<double>(gy, h->axy.d, h->w1, h->w1, 1, nullptr, h->stream));
  }
  if (h->precision == IB_PREC_MIXED) {
    df64* w2 = view<df64>(h->w2);
    if (h->fx_solve) {
      CK(poisson_fx<df64>(h, w2, w2, 1, view<df64>(h->rings), op_lap(h), nullptr, h->w1));
      CK(poisson_fx<df64>(h, w2, w2, 1, nullptr, op_cn1(h), w2, h->w1));
    }
    for (int sw = 1; sw <= h->refine; ++sw) {
      CK(poisson_mixed(h, w2, w2, 1, view<df64>(h->rings), op_lap(h), nullptr, h->w32, h->x032, h->x132, sw));
      CK(poisson_mixed(h, w2, w2, 1, nullptr, op_cn1(h), w2, h->w32, h->x032, h->x132, sw));
    }
  }
  CK(cudaMemsetAsync(h->w1, 0, sizeof(double) * g.nlev * g.nG, h->stream));
  CK(cudaMemsetAsync(h->w2, 0, sizeof(double) * g.nlev * g.nG, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return IB_OK;
}

int capture_graphs(ib_handle* h) {
  ib::Range nvtx_range("capture step graphs");
  for (int p = 0; p < 2; ++p) {
    if (h->gexec[p]) { cudaGraphExecDestroy(h->gexec[p]); h->gexec[p] = nullptr; }
    cudaGraph_t graph = nullptr;
    CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    g_pdl = h->use_pdl;  // kernels of the static step overlap their launch with the predecessor's tail
    cudaError_t e = enqueue_step_mode(h, p);
    g_pdl = false;
    cudaError_t e2 = cudaStreamEndCapture(h->stream, &graph);
    if (e != cudaSuccess) { if (graph) cudaGraphDestroy(graph); return fail(h, IB_ERR_CUDA, "step capture", e); }
    if (e2 != cudaSuccess) return fail(h, IB_ERR_CUDA, "step capture", e2);
    size_t nn = 0;
    if (cudaGraphGetNodes(graph, nullptr, &nn) == cudaSuccess && nn > 0) {
      std::vector<cudaGraphNode_t> nodes(nn);
      cudaGraphGetNodes(graph, nodes.data(), &nn);
      int k = 0;
      for (auto nd : nodes) {
        cudaGraphNodeType ty;
        if (cudaGraphNodeGetType(nd, &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel) ++k;
      }
      h->kernels_per_step = k;
    }
    e = cudaGraphInstantiate(&h->gexec[p], graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "graph instantiate", e);
  }
  return IB_OK;
}

void destroy_handle(ib_handle* h) {
  if (!h) return;
  DeviceGuard dev_guard_(h->device >= 0 ? h->device : 0);
  if (h->stream) cudaStreamSynchronize(h->stream);
  for (auto& ge : h->gexec)
    if (ge) cudaGraphExecDestroy(ge);
  for (auto& ge : h->mgexec)
    if (ge) cudaGraphExecDestroy(ge);
  if (h->h_mslot) cudaFreeHost(h->h_mslot);
  for (double* b : {h->asm_G, h->asm_P, h->asm_Wa, h->asm_Wb, h->asm_Q, h->asm_R, h->asm_work})
    if (b) cudaFree(b);
  if (h->h_cgout) cudaFreeHost(h->h_cgout);
  if (h->loop_stream) cudaStreamDestroy(h->loop_stream);
  for (void* p : h->allocs) cudaFree(p);
  if (h->op_work) cudaFree(h->op_work);
  if (h->h_q0) cudaFreeHost(h->h_q0);
  if (h->status) cudaFreeHost(h->status);
  if (h->h_stress) cudaFreeHost(h->h_stress);
  if (h->h_sc) cudaFreeHost(h->h_sc);
  delete h->mlp;
  h->axx.release();
  h->axy.release();
  h->axx32.release();
  h->axy32.release();
  h->sgx.release();
  h->sgy.release();
  h->rplan.release();
  for (auto ev : h->fork_ev)
    if (ev) cudaEventDestroy(ev);
  for (auto ev : h->stress_ev)
    if (ev) cudaEventDestroy(ev);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

int stage_q0(ib_handle* h, double u, double v, const double* kin = nullptr) {
  const int L = h->g.nlev;
  const int slot_len = 2 * L + 6 * h->nbodies;
  if (h->q0_slot >= kQ0Slots) {
    CK(cudaStreamSynchronize(h->stream));
    h->q0_slot = 0;
  }
  double* slot = h->h_q0 + (size_t)h->q0_slot * slot_len;
  h->q0_slot++;
  for (int l = 0; l < L; ++l) {
    const double hc = h->g.h * std::ldexp(1.0, l);  // gridstep(grid, lev), fluids.jl:102
    slot[2 * l] = u * hc;                            // base_flux!, fluid-ops.jl:414-415
    slot[2 * l + 1] = v * hc;
  }
  CK(cudaMemcpyAsync(h->d_q0, slot, sizeof(double) * 2 * L, cudaMemcpyHostToDevice, h->stream));
  if (kin && h->motion == IB_MOTION_PRESCRIBED) {
    std::memcpy(slot + 2 * L, kin, sizeof(double) * 6 * h->nbodies);
    CK(cudaMemcpyAsync(h->d_kin, slot + 2 * L, sizeof(double) * 6 * h->nbodies, cudaMemcpyHostToDevice, h->stream));
  }
  return IB_OK;
}

// Conjugate gradients for B Fb = ftmp (cg!(qty.Fb, B, ftmp), cnab/ops.jl:104-114), warm-started
// from h->fb, stopping when ||r|| <= tol ||ftmp||.  The residual norm is read back each iteration.
// The CG vectors are FP64 in both modes; S is the state type of the B products.
//
// With a preconditioner (IB_PC_SCHUR_REF) this is PCG with z = P r, P the inverse Schur matrix of
// a reference configuration (row-major h->binv_rm); the stopping rule is unchanged.
// Scalars: sc[0] = r.z, sc[1] = p.Ap, sc[2] = new r.z, sc[3] = rhs.rhs, sc[4] = r.r.
template <typename S>
int cg_solve(ib_handle* h) {
  ib::Range nvtx_range("CG solve");
  const int nf = h->nf;
  cudaStream_t s = h->stream;
  double *x = h->fb, *r = h->cg_r, *p = h->cg_p, *Ap = h->cg_Ap, *sc = h->cg_sc;
  const bool pc = h->precond == IB_PC_SCHUR_REF && h->binv_rm && h->pc_step >= 0;
  double* z = pc ? h->cg_z : r;
  CK(schur_apply<S>(h, x, Ap));
  CK(cudaMemcpyAsync(r, h->ftmp, sizeof(double) * nf, cudaMemcpyDeviceToDevice, s));
  CK(vec_axpy(r, Ap, -1.0, nf, s));
  CK(vec_dot(r, r, nf, sc + 4, s));
  CK(vec_dot(h->ftmp, h->ftmp, nf, sc + 3, s));
  if (pc) CK(gemv_rowmajor(h->binv_rm, r, z, nf, s));
  CK(vec_dot(r, z, nf, sc + 0, s));
  CK(cudaMemcpyAsync(p, z, sizeof(double) * nf, cudaMemcpyDeviceToDevice, s));
  CK(cudaMemcpyAsync(h->h_sc, sc, sizeof(double) * 5, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  const double target = h->cg_tol * std::sqrt(h->h_sc[3]);
  double rn = std::sqrt(h->h_sc[4]);
  if (!std::isfinite(rn)) return fail(h, IB_ERR_NONFINITE, "infinite flux");
  h->cg_res0.push_back(h->h_sc[3] > 0 ? rn / std::sqrt(h->h_sc[3]) : rn);
  int it = 0;
  bool conv = rn <= target;
  const auto t_loop = std::chrono::steady_clock::now();
  while (!conv && it < h->cg_maxiter) {
    ++it;
    CK(schur_apply<S>(h, p, Ap));
    CK(vec_dot(p, Ap, nf, sc + 1, s));
    CK(cg_update_xr(x, r, p, Ap, sc, nf, s));
    CK(vec_dot(r, r, nf, sc + 4, s));
    CK(cudaMemcpyAsync(h->h_sc + 4, sc + 4, sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    rn = std::sqrt(h->h_sc[4]);
    if (!std::isfinite(rn)) return fail(h, IB_ERR_NONFINITE, "infinite flux");
    conv = rn <= target;
    if (!conv) {
      if (pc) {
        CK(gemv_rowmajor(h->binv_rm, r, z, nf, s));
        CK(vec_dot(r, z, nf, sc + 2, s));
      } else {
        CK(vec_dot(r, r, nf, sc + 2, s));
      }
      CK(cg_update_p(p, z, sc, nf, s));
    }
  }
  if (it > 0) {
    const double per = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_loop).count() / it;
    h->cg_iter_s = h->cg_iter_s > 0.0 ? 0.9 * h->cg_iter_s + 0.1 * per : per;
  }
  h->cg_iters.push_back(it);
  h->cg_res.push_back(h->h_sc[3] > 0 ? rn / std::sqrt(h->h_sc[3]) : rn);
  if (!conv) return fail(h, IB_ERR_CG_MAXITER, "Schur CG reached its iteration cap");
  return IB_OK;
}

// The training's blend minimises the held-out force error in the 2-norm.  The CG start residual
// is that error times the Schur operator B (condition number ~1e4-1e5), which amplifies a
// correction that is rough from point to point, so a blend that barely lowers the 2-norm error
// can raise ||B x0 - rhs||.  This re-fits the blend in the norm CG sees: over the most recent
// held-out rows j (at most 256), blend = argmin over [0, 1] of sum_j |B (blend q_j - t_j)|^2,
// with q_j the network's correction, t_j the extrapolation's error and B the operator of the
// current configuration.  The B products run on the Schur scratch arrays; the two a later
// product starts from (Pw, rings_w: the previous call's psi and rings) are saved and restored,
// so the run's later CG iterates are those it would have had without this validation, and so
// are the status flags (a non-finite network correction would otherwise leave the handle's
// "infinite flux" flag set; its rows make the blend 0 instead).
template <typename S>
int learn_validate_schur(ib_handle* h) {
  learn::Mlp& m = *h->mlp;
  const int nf = h->nf;
  const Geometry& g = h->g;
  cudaStream_t s = h->stream;
  constexpr int kRows = 256;
  const size_t npw = (size_t)g.nlev * g.nG, nrw = (size_t)g.nlev * g.nbc;  // 8-byte elements either way
  double *q = nullptr, *t = nullptr, *bq = nullptr, *bt = nullptr, *dots = nullptr, *save = nullptr;
  auto release = [&]() {
    for (double* p : {q, t, bq, bt, dots, save})
      if (p) cudaFree(p);
  };
  auto al = [&](double** p, size_t n) { return cudaMalloc(p, sizeof(double) * std::max<size_t>(n, 1)); };
  cudaError_t e;
  if ((e = al(&q, (size_t)kRows * nf)) != cudaSuccess || (e = al(&t, (size_t)kRows * nf)) != cudaSuccess ||
      (e = al(&bq, nf)) != cudaSuccess || (e = al(&bt, nf)) != cudaSuccess || (e = al(&dots, 3 * kRows)) != cudaSuccess ||
      (e = al(&save, npw + nrw + 2)) != cudaSuccess) {
    release();
    return fail(h, IB_ERR_CUDA, "learned-start validation buffers", e);
  }
  int rows = 0;
  int* status_save = reinterpret_cast<int*>(save + npw + nrw);  // the 4 status flags
  e = m.heldout(q, t, kRows, &rows);
  if (e == cudaSuccess) e = cudaMemcpyAsync(status_save, h->status, 4 * sizeof(int), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(save, h->Pw, sizeof(double) * npw, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(save + npw, h->rings_w, sizeof(double) * nrw, cudaMemcpyDeviceToDevice, s);
  for (int j = 0; j < rows && e == cudaSuccess; ++j) {
    if ((e = schur_apply<S>(h, q + (size_t)j * nf, bq)) != cudaSuccess) break;
    if ((e = schur_apply<S>(h, t + (size_t)j * nf, bt)) != cudaSuccess) break;
    if ((e = vec_dot(bq, bt, nf, dots + 3 * j, s)) != cudaSuccess) break;
    if ((e = vec_dot(bq, bq, nf, dots + 3 * j + 1, s)) != cudaSuccess) break;
    e = vec_dot(bt, bt, nf, dots + 3 * j + 2, s);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->Pw, save, sizeof(double) * npw, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->rings_w, save + npw, sizeof(double) * nrw, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->status, status_save, 4 * sizeof(int), cudaMemcpyDeviceToHost, s);
  std::vector<double> hd(3 * (size_t)std::max(rows, 1));
  if (e == cudaSuccess && rows > 0)
    e = cudaMemcpyAsync(hd.data(), dots, sizeof(double) * 3 * rows, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  release();
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "learned-start validation", e);
  if (rows == 0) return check_status(h);
  double tq = 0.0, qq = 0.0, tt = 0.0;
  for (int j = 0; j < rows; ++j) {
    tq += hd[3 * j];
    qq += hd[3 * j + 1];
    tt += hd[3 * j + 2];
  }
  if (!std::isfinite(tq) || !std::isfinite(qq)) {
    m.blend = 0.0;
    m.val_rel = 1.0;
  } else {
    m.blend = qq > 0.0 ? std::min(1.0, std::max(0.0, tq / qq)) : 0.0;
    m.val_rel = tt > 0.0 ? (tt - 2.0 * m.blend * tq + m.blend * m.blend * qq) / tt : 0.0;
  }
  return check_status(h);
}

// warm start (h->fb holds F_{n-1}, h->fb_prev F_{n-2}): the previous Fb (the reference's cg! on
// qty.Fb), its linear extrapolation, zero, or the learned prediction (extrapolation until a
// network is trained); keeps F_{n-1} in h->fb_last and the network's features
cudaError_t enqueue_warm_start(ib_handle* h, bool hist2) {
  cudaStream_t s = h->stream;
  const size_t fbytes = sizeof(double) * h->nf;
  CE(cudaMemcpyAsync(h->fb_last, h->fb, fbytes, cudaMemcpyDeviceToDevice, s));
  const bool use_mlp = h->mlp && (h->collect || h->warm_start == IB_WARM_LEARNED);
  if (use_mlp) CE(h->mlp->features(h->d_kin, 6 * h->nbodies, h->fb_last, h->fb_prev, h->nf));
  switch (h->warm_start) {
    case IB_WARM_ZERO: CE(cudaMemsetAsync(h->fb, 0, fbytes, s)); break;
    case IB_WARM_EXTRAPOLATE:
      if (hist2) CE(axpby<double>(h->fb, h->fb_prev, -1.0, 2.0, h->nf, s));
      break;
    case IB_WARM_LEARNED:
      if (hist2 && h->mlp && h->mlp->trained) CE(h->mlp->predict(h->fb_last, h->fb_prev, h->fb));
      else if (hist2) CE(axpby<double>(h->fb, h->fb_prev, -1.0, 2.0, h->nf, s));
      break;
    default: break;
  }
  return cudaSuccess;
}

// preconditioner: the inverse Schur matrix of the current configuration, assembled at the first
// step and again every pc_refresh steps, or (pc_refresh = 0) once the iterations spent above
// those of the first solve after the last assembly have cost as much time as an assembly
int pc_maybe_assemble(ib_handle* h) {
  if (h->precond != IB_PC_SCHUR_REF) return IB_OK;
  const bool due = h->pc_step < 0 ||
                   (h->pc_refresh > 0 ? h->steps - h->pc_step >= h->pc_refresh
                                      : h->pc_excess_iters * h->cg_iter_s >= h->pc_assembly_s);
  if (!due) return IB_OK;
  const auto t_asm = std::chrono::steady_clock::now();
  if (!h->bmat) {
    const int64_t n2 = (int64_t)h->nf * h->nf;
    CK(h->alloc(&h->bmat, n2));
    CK(h->alloc(&h->binv_cm, n2));
    CK(h->alloc(&h->binv_rm, n2));
  }
  int rc = assemble_schur(h);
  if (rc != IB_OK) return rc;
  rc = check_status(h);
  if (rc != IB_OK) return rc;
  h->pc_step = h->steps;
  h->pc_base_iters = -1;
  h->pc_excess_iters = 0.0;
  h->pc_assemblies++;
  h->pc_assembly_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t_asm).count();
  return IB_OK;
}

// the first solve after an assembly starts at the previous Fb of a changed matrix; the second
// one (solve_step > pc_step) sets the base for the extra-iteration count
void pc_account(ib_handle* h, int64_t solve_step) {
  if (h->precond != IB_PC_SCHUR_REF || h->cg_iters.empty()) return;
  const int it_now = h->cg_iters.back();
  if (h->pc_base_iters < 0 && solve_step > h->pc_step) h->pc_base_iters = it_now;
  else if (h->pc_base_iters >= 0) h->pc_excess_iters += std::max(0, it_now - h->pc_base_iters);
}

// advance! for rigidly moving bodies (corrected reference branch): points and weights from the
// step's kinematics, the trial state, Fb by CG, stress, projection and Vort2Flux.
template <typename S>
int moving_step(ib_handle* h, double t, double u, double v, const double* kin) {
  ib::Range nvtx_range("moving step");
  const Geometry& g = h->g;
  cudaStream_t s = h->stream;
  const int p = h->parity;
  int rc = stage_q0(h, u, v, kin);
  if (rc != IB_OK) return rc;
  // a/b. update_bodies! and update!(reg, points)
  CK(body_points(h->xb_body, h->d_kin, h->body_of, h->nb, h->xb, h->vb, s));
  CK(reg_update(g, h->xb, h->nb, h->body_idx, h->weight, h->status, s));
  CK(enqueue_trial<S>(h, p));
  // e. BoundaryForcer for moving bodies (timestepping.jl:122-139): ftmp = E(qs + q0) - ub h
  CK(reg_gather<S>(g, view<S>(h->qs1), h->d_q0, h->body_idx, h->weight, h->nb, h->ftmp, 1, g.nq, h->nf, s));
  CK(vec_axpy(h->ftmp, h->vb, -g.h, h->nf, s));
  rc = check_status(h);
  if (rc != IB_OK) return rc;
  const bool hist2 = h->steps >= 2;
  CK(enqueue_warm_start(h, hist2));
  rc = pc_maybe_assemble(h);
  if (rc != IB_OK) return rc;
  rc = cg_solve<S>(h);
  if (rc != IB_OK) return rc;
  pc_account(h, h->steps);
  if (h->mlp && h->collect && hist2) CK(h->mlp->record(h->fb));
  CK(cudaMemcpyAsync(h->fb_prev, h->fb_last, sizeof(double) * h->nf, cudaMemcpyDeviceToDevice, s));
  CK(enqueue_stress(h));
  CK(enqueue_project<S>(h, p));
  h->parity ^= 1;
  h->steps++;
  h->t = t;
  return check_status(h);
}

// ---- the moving step as a captured graph (steps >= 2) -------------------------------------------
// Per parity one graph: staging copies of the base flux and kinematics from a pinned slot, the
// body update, trial state, forcing, warm start, CG with a device-side convergence test (a
// while-conditional node), stress, projection and Vort2Flux, and copies of the CG statistics and
// status flags to pinned memory.  The host launches it, waits, and keeps the statistics, the
// preconditioner policy and the error reporting of the eager step.

// Records the moving step for buffer parity p into the capture h->stream belongs to (its own,
// or an ensemble's that it joined); `k` is the step's index within a multi-step launch, which
// selects its pinned staging slot and statistics record.
template <typename S>
cudaError_t enqueue_moving_captured(ib_handle* h, int p, int k = 0) {
  const Geometry& g = h->g;
  cudaStream_t s = h->stream;
  const int L = g.nlev;
  const double* slot = h->h_mslot + (size_t)k * (2 * L + 6 * h->nbodies);
  double* cgout = h->h_cgout + 4 * k;
  const size_t fbytes = sizeof(double) * h->nf;
  const bool pc = h->precond == IB_PC_SCHUR_REF && h->binv_rm;
  double *x = h->fb, *r = h->cg_r, *pv = h->cg_p, *Ap = h->cg_Ap, *sc = h->cg_sc;
  double* z = pc ? h->cg_z : r;
  auto body = [&]() -> cudaError_t {
    CE(cudaMemcpyAsync(h->d_q0, slot, sizeof(double) * 2 * L, cudaMemcpyHostToDevice, s));
    CE(cudaMemcpyAsync(h->d_kin, slot + 2 * L, sizeof(double) * 6 * h->nbodies, cudaMemcpyHostToDevice, s));
    CE(body_points(h->xb_body, h->d_kin, h->body_of, h->nb, h->xb, h->vb, s));
    CE(reg_update(g, h->xb, h->nb, h->body_idx, h->weight, h->status, s));
    CE(enqueue_trial<S>(h, p));
    CE(reg_gather<S>(g, view<S>(h->qs1), h->d_q0, h->body_idx, h->weight, h->nb, h->ftmp, 1, g.nq, h->nf, s));
    CE(vec_axpy(h->ftmp, h->vb, -g.h, h->nf, s));
    CE(enqueue_warm_start(h, true));
    // CG start (as cg_solve)
    CE(schur_apply<S>(h, x, Ap));
    CE(cudaMemcpyAsync(r, h->ftmp, fbytes, cudaMemcpyDeviceToDevice, s));
    CE(vec_axpy(r, Ap, -1.0, h->nf, s));
    CE(vec_dot(r, r, h->nf, sc + 4, s));
    CE(vec_dot(h->ftmp, h->ftmp, h->nf, sc + 3, s));
    if (pc) CE(gemv_rowmajor(h->binv_rm, r, z, h->nf, s));
    CE(vec_dot(r, z, h->nf, sc + 0, s));
    CE(cudaMemcpyAsync(pv, z, fbytes, cudaMemcpyDeviceToDevice, s));
    // while-conditional node: the loop body is captured on the side stream into its graph
    cudaStreamCaptureStatus cs;
    cudaGraph_t cg = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    const cudaGraphEdgeData* edges = nullptr;
    size_t ndeps = 0;
    CE(cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, &deps, &edges, &ndeps));
    cudaGraphConditionalHandle cond;
    CE(cudaGraphConditionalHandleCreate(&cond, cg, 0, cudaGraphCondAssignDefault));
    CE(cg_start(sc, h->d_cgctl, h->cg_tol, h->status, h->d_cgout, cond, s));
    CE(cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, &deps, &edges, &ndeps));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    CE(cudaGraphAddNode(&node, cg, deps, edges, ndeps, &cp));
    cudaGraph_t loop = cp.conditional.phGraph_out[0];
    CE(cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    cudaStream_t ls = h->loop_stream;
    CE(cudaStreamBeginCaptureToGraph(ls, loop, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    h->stream = ls;
    cudaError_t le = [&]() -> cudaError_t {
      CE(schur_apply<S>(h, pv, Ap));
      CE(vec_dot(pv, Ap, h->nf, sc + 1, ls));
      CE(cg_update_xr(x, r, pv, Ap, sc, h->nf, ls));
      CE(vec_dot(r, r, h->nf, sc + 4, ls));
      if (pc) CE(gemv_rowmajor(h->binv_rm, r, z, h->nf, ls));
      CE(vec_dot(r, z, h->nf, sc + 2, ls));
      CE(cg_update_p(pv, z, sc, h->nf, ls));
      return cg_check(sc, h->d_cgctl, h->cg_maxiter, h->status, cond, ls);
    }();
    h->stream = s;
    cudaGraph_t loop_out = nullptr;
    cudaError_t le2 = cudaStreamEndCapture(ls, &loop_out);
    CE(le);
    CE(le2);
    CE(cg_finish(sc, h->d_cgctl, h->d_cgout, s));
    if (h->mlp && h->collect) CE(h->mlp->record_enqueue(h->fb));
    CE(cudaMemcpyAsync(h->fb_prev, h->fb_last, fbytes, cudaMemcpyDeviceToDevice, s));
    CE(enqueue_stress(h));
    CE(enqueue_project<S>(h, p));
    CE(cudaMemcpyAsync(cgout, h->d_cgout, sizeof(double) * 4, cudaMemcpyDeviceToHost, s));
    return cudaSuccess;
  };
  cudaError_t e = body();
  h->stream = s;
  return e;
}

template <typename S>
int capture_moving(ib_handle* h, int p) {
  cudaStream_t s = h->stream;
  cudaGraph_t graph = nullptr;
  CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  cudaError_t e = enqueue_moving_captured<S>(h, p);
  cudaError_t e2 = cudaStreamEndCapture(s, &graph);
  if (e != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    return fail(h, IB_ERR_CUDA, "moving-step capture", e);
  }
  if (e2 != cudaSuccess) return fail(h, IB_ERR_CUDA, "moving-step capture", e2);
  if (h->mgexec[p]) {
    cudaGraphExecDestroy(h->mgexec[p]);
    h->mgexec[p] = nullptr;
  }
  e = cudaGraphInstantiate(&h->mgexec[p], graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "moving-step graph instantiate", e);
  return IB_OK;
}

// what the captured moving step depends on besides the device buffers
uint64_t moving_graph_key(const ib_handle* h) {
  uint64_t k = (uint64_t)h->warm_start;
  k = k * 31 + (uint64_t)h->precond;
  k = k * 31 + (uint64_t)(h->binv_rm != nullptr);
  k = k * 31 + (uint64_t)(h->mlp != nullptr);
  k = k * 31 + (uint64_t)h->collect;
  k = k * 31 + (uint64_t)(h->mlp && h->mlp->trained);
  k = k * 31 + (uint64_t)h->cg_maxiter;
  uint64_t tb;
  std::memcpy(&tb, &h->cg_tol, sizeof(tb));
  k = k * 31 + tb;
  return k;
}

template <typename S>
int moving_step_graph(ib_handle* h, double t, double u, double v, const double* kin) {
  ib::Range nvtx_range("moving step (graph)");
  const Geometry& g = h->g;
  // base flux and kinematics of this step into the pinned slot the graphs copy from (the
  // previous launch is complete: every step ends with a synchronisation)
  for (int l = 0; l < g.nlev; ++l) {
    const double hc = g.h * std::ldexp(1.0, l);  // base_flux!, fluid-ops.jl:414-415
    h->h_mslot[2 * l] = u * hc;
    h->h_mslot[2 * l + 1] = v * hc;
  }
  std::memcpy(h->h_mslot + 2 * g.nlev, kin, sizeof(double) * 6 * h->nbodies);
  int rc = pc_maybe_assemble(h);
  if (rc != IB_OK) return rc;
  const uint64_t key = moving_graph_key(h);
  if (!h->mgexec[0] || key != h->mg_key) {
    for (int p = 0; p < 2; ++p) {
      rc = capture_moving<S>(h, p);
      if (rc != IB_OK) return rc;
    }
    h->mg_key = key;
  }
  CK(cudaGraphLaunch(h->mgexec[h->parity], h->stream));
  CK(cudaStreamSynchronize(h->stream));
  const double* o = h->h_cgout;
  h->cg_iters.push_back((int)o[0]);
  h->cg_res.push_back(o[1]);
  h->cg_res0.push_back(o[2]);
  if (h->mlp && h->collect) h->mlp->record_commit();
  pc_account(h, h->steps);
  h->parity ^= 1;
  h->steps++;
  h->t = t;
  rc = check_status(h);
  if (rc != IB_OK) return rc;
  if (o[3] != 0.0) return fail(h, IB_ERR_CG_MAXITER, "Schur CG reached its iteration cap");
  return IB_OK;
}

int moving_step_mode(ib_handle* h, double t, double u, double v, const double* kin) {
  // the first two steps (no force history yet, first preconditioner) run eagerly
  const bool graph = h->use_moving_graph && h->steps >= 2 && (h->precond != IB_PC_SCHUR_REF || h->pc_step >= 0);
  if (h->precision == IB_PREC_MIXED)
    return graph ? moving_step_graph<df64>(h, t, u, v, kin) : moving_step<df64>(h, t, u, v, kin);
  return graph ? moving_step_graph<double>(h, t, u, v, kin) : moving_step<double>(h, t, u, v, kin);
}

// ---- setup-time autotuner ---------------------------------------------------------------------
// Chooses, by timing on this GPU, the transform form of the solves (Stockham FFT passes, warp-per-
// line FFT passes, or BF16x3 tensor-core GEMMs for mixed precision) and, for mixed precision on
// warp passes, the Vort2Flux order (all levels in one batch, or level by level).  The timed unit
// is the transform work a step repeats: the batched Crank-Nicolson solve over all levels, a
// projection-size solve, a full Vort2Flux and a level-1-only Vort2Flux, run on scratch arrays
// (the state is not touched); the stencil, body and Schur kernels are the same for every
// candidate.  Each candidate runs once to warm up, then five times in each of three rounds; the
// fastest run counts.
// IBGB300_DST / IBGB300_V2F pin a choice, IBGB300_AUTOTUNE=0 keeps the fixed size rules.
template <typename S>
cudaError_t tune_unit(ib_handle* h, double* gam, double* psi, double* q, double* q1, double* rings, double* in,
                      double* out) {
  const int L = h->g.nlev;
  CE(solve(h, view<S>(in), view<S>(out), L, nullptr, op_cn_all(h), nullptr));
  CE(solve(h, view<S>(in), view<S>(out), 1, nullptr, op_cn1(h), view<S>(out)));
  CE(vort2flux<S>(h, view<S>(gam), view<S>(psi), view<S>(q), nullptr, view<S>(rings)));
  return vort2flux<S>(h, view<S>(gam), view<S>(psi), nullptr, view<S>(q1), view<S>(rings));
}

double tune_time(ib_handle* h, double* gam, double* psi, double* q, double* q1, double* rings, double* in, double* out) {
  cudaStream_t s = h->stream;
  auto run = [&]() {
    return h->precision == IB_PREC_MIXED ? tune_unit<df64>(h, gam, psi, q, q1, rings, in, out)
                                         : tune_unit<double>(h, gam, psi, q, q1, rings, in, out);
  };
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return -1.0;
  double best = -1.0;
  bool ok = run() == cudaSuccess && cudaStreamSynchronize(s) == cudaSuccess;
  for (int r = 0; ok && r < 5; ++r) {
    float ms = 0.0f;
    ok = cudaEventRecord(e0, s) == cudaSuccess && run() == cudaSuccess && cudaEventRecord(e1, s) == cudaSuccess &&
         cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess;
    if (ok && (best < 0 || ms < best)) best = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!ok) {
    cudaGetLastError();  // a candidate that cannot run is skipped
    cudaStreamSynchronize(s);
    return -1.0;
  }
  return best;
}

// Decisions are kept per process for each (device, grid, levels, sweeps, what is tuned), so every
// handle of one shape in a process (an ensemble member and the same problem stepped alone, say)
// takes the same choice and gives the same bits.
struct TuneRecord {
  double ms[12];
  int best;
};
std::mutex g_tune_mu;
std::map<std::string, TuneRecord> g_tune_cache;

int autotune(ib_handle* h, bool tune_form, bool tune_v2f, bool lv_base) {
  ib::Range nvtx_range("autotune");
  const Geometry& g = h->g;
  const int L = g.nlev;
  char keybuf[160];
  std::snprintf(keybuf, sizeof(keybuf), "%d/%d/%d/%d/%d/%d/%d/%d/%d/%d", h->device, g.nx, g.ny, L, h->precision, h->refine,
                (int)tune_form, (int)tune_v2f, (int)h->wdst, (int)h->gdst);
  const std::string key(keybuf);
  std::lock_guard<std::mutex> tune_lock(g_tune_mu);
  const auto hit = g_tune_cache.find(key);
  const bool mixed = h->precision == IB_PREC_MIXED;
  const bool wsup = wdst_axis_supported(g.nx) && wdst_axis_supported(g.ny);
  const bool tsup = mixed && sgemm_axis_supported(g.nx) && sgemm_axis_supported(g.ny);
  std::vector<void*> tmp;
  const bool timing = hit == g_tune_cache.end();
  auto scratch = [&](size_t n) -> double* {
    if (!timing) return reinterpret_cast<double*>(16);  // unused: the choice is known
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(double) * (n > 0 ? n : 1)) != cudaSuccess) return nullptr;
    cudaMemset(p, 0, sizeof(double) * (n > 0 ? n : 1));
    tmp.push_back(p);
    return static_cast<double*>(p);
  };
  const int64_t nG = g.nG;
  double* gam = scratch(L * nG);
  double* psi = scratch(L * nG);
  double* q = scratch((int64_t)L * g.nq);
  double* q1 = scratch(g.nq);
  double* rings = scratch((int64_t)L * g.nbc);
  double* in = scratch(L * nG);
  double* out = scratch(L * nG);
  auto release = [&]() {
    for (void* p : tmp) cudaFree(p);
  };
  if (!gam || !psi || !q || !q1 || !rings || !in || !out) {
    release();
    return fail(h, IB_ERR_CUDA, "autotuner scratch allocation");
  }
  const bool wdst0 = h->wdst, gdst0 = h->gdst, lv0 = h->v2f_levels, fx0 = h->fx_solve;
  h->fx_solve = h->v2f_fx = false;  // the candidates are the FP32 passes
  struct Cand { int form; bool levels; bool yalt; };
  std::vector<Cand> cands;
  std::vector<int> forms;
  if (tune_form) {
    forms.push_back(IB_FORM_STOCKHAM);
    if (wsup) forms.push_back(IB_FORM_WARP);
    if (tsup) forms.push_back(IB_FORM_TENSOR);
  } else {
    forms.push_back(h->gdst ? IB_FORM_TENSOR : (h->wdst ? IB_FORM_WARP : IB_FORM_STOCKHAM));
  }
  for (int f : forms) {
    const bool lv_ok = mixed && lv_base && f == IB_FORM_WARP;
    // the warp y pass has a second compiled occupancy (8 blocks per SM) to try
    const int ny_alt = (mixed && f == IB_FORM_WARP && IB_WDST_YMINB != 8) ? 2 : 1;
    for (int ya = 0; ya < ny_alt; ++ya) {
      if (tune_v2f) {
        cands.push_back({f, false, ya == 1});
        if (lv_ok) cands.push_back({f, true, ya == 1});
      } else {
        cands.push_back({f, lv0 && lv_ok, ya == 1});
      }
    }
  }
  bool need_tc = false, need_lv = false;
  if (hit != g_tune_cache.end()) {
    need_tc = hit->second.best / 4 == IB_FORM_TENSOR;
    need_lv = (hit->second.best / 2) % 2 != 0;
  } else {
    for (const Cand& c : cands) {
      need_tc |= c.form == IB_FORM_TENSOR;
      need_lv |= c.levels;
    }
  }
  cudaError_t e;
  const bool tc_own = need_tc && !h->gw32;  // the tensor-core resources are the tuner's to keep or free
  if (tc_own) {
    if ((e = h->sgx.build(g.nx)) != cudaSuccess || (e = h->sgy.build(g.ny)) != cudaSuccess) {
      release();
      return fail(h, IB_ERR_CUDA, "sine-matrix image", e);
    }
    void* p = nullptr;
    if ((e = cudaMalloc(&p, sizeof(float) * L * nG)) != cudaSuccess) {
      release();
      return fail(h, IB_ERR_CUDA, "autotuner work allocation", e);
    }
    h->gw32 = static_cast<float*>(p);
  }
  if (need_lv && !h->rplan.St) {
    if ((e = h->rplan.build(g, h->mLap)) != cudaSuccess) {
      release();
      return fail(h, IB_ERR_CUDA, "ring transfer tables", e);
    }
  }
  int best = -1;
  double best_ms = -1.0;
  if (hit != g_tune_cache.end()) {
    best = hit->second.best;
    for (int i = 0; i < 12; ++i) h->tune_ms[i] = hit->second.ms[i];
  } else {
    // three interleaved rounds (so a clock ramp or a neighbour's burst does not favour one
    // candidate), the fastest of each candidate's 15 runs counts
    for (int round = 0; round < 3; ++round)
      for (const Cand& c : cands) {
        h->wdst = c.form == IB_FORM_WARP;
        h->gdst = c.form == IB_FORM_TENSOR;
        h->v2f_levels = c.levels;
        h->axy32.d.wMinB = c.yalt ? 8 : IB_WDST_YMINB;
        const double ms = tune_time(h, gam, psi, q, q1, rings, in, out);
        const int idx = (c.form * 2 + (c.levels ? 1 : 0)) * 2 + (c.yalt ? 1 : 0);
        if (ms > 0 && (h->tune_ms[idx] < 0 || ms < h->tune_ms[idx])) h->tune_ms[idx] = ms;
      }
    // the fastest, unless the size rule's choice is within 1% of it (timing noise)
    const int rule = ((gdst0 ? IB_FORM_TENSOR : (wdst0 ? IB_FORM_WARP : IB_FORM_STOCKHAM)) * 2 + (lv0 ? 1 : 0)) * 2;
    for (int i = 0; i < 12; ++i)
      if (h->tune_ms[i] > 0 && (best < 0 || h->tune_ms[i] < best_ms)) {
        best = i;
        best_ms = h->tune_ms[i];
      }
    if (best >= 0 && h->tune_ms[rule] > 0 && h->tune_ms[rule] <= 1.01 * best_ms) best = rule;
    if (best >= 0) {
      TuneRecord rec;
      for (int i = 0; i < 12; ++i) rec.ms[i] = h->tune_ms[i];
      rec.best = best;
      g_tune_cache[key] = rec;
    }
  }
  release();
  h->fx_solve = fx0;
  if (best < 0) {
    h->wdst = wdst0;
    h->gdst = gdst0;
    h->v2f_levels = lv0;
    h->axy32.d.wMinB = IB_WDST_YMINB;
  } else {
    h->wdst = best / 4 == IB_FORM_WARP;
    h->gdst = best / 4 == IB_FORM_TENSOR;
    h->v2f_levels = (best / 2) % 2 != 0;
    h->axy32.d.wMinB = (best % 2) ? 8 : IB_WDST_YMINB;
  }
  // keep what the choice uses: the tensor-core tables and work array, the ring-transfer plan
  if (tc_own && !h->gdst) {
    cudaFree(h->gw32);
    h->gw32 = nullptr;
    h->sgx.release();
    h->sgy.release();
  } else if (tc_own) {
    h->allocs.push_back(h->gw32);
    h->device_bytes += (int64_t)sizeof(float) * L * nG;
  }
  if (!h->v2f_levels && h->rplan.St) h->rplan.release();
  h->tuned = best >= 0;
  return cudaGetLastError() == cudaSuccess ? IB_OK : fail(h, IB_ERR_CUDA, "autotuner");
}

int one_step(ib_handle* h, double t, double u, double v) {
  if (h->motion == IB_MOTION_PRESCRIBED) return fail(h, IB_ERR_INVALID, "moving bodies need kinematics (ib_advance_kin)");
  int rc = stage_q0(h, u, v);
  if (rc != IB_OK) return rc;
  if (h->use_graph) {
    CK(cudaGraphLaunch(h->gexec[h->parity], h->stream));
  } else {
    CK(enqueue_step_mode(h, h->parity));
  }
  h->parity ^= 1;
  h->steps++;
  h->t = t;
  return IB_OK;
}

}  // namespace

bool ib_handle_lap_view(const ib_handle* h, ib::LapView* v) {
  if (!h || !v) return false;
  v->g = h->g;
  v->ax = h->axx.d;
  v->ay = h->axy.d;
  v->mlap = h->mLap;
  v->stream = h->stream;
  v->device = h->device;
  return true;
}

int ib_handle_fail(ib_handle* h, int code, const char* msg) { return fail(h, code, msg); }

// ================================================================================================
// C ABI
// ================================================================================================
extern "C" {

const char* ib_status_string(int status) {
  switch (status) {
    case IB_OK: return "ok";
    case IB_ERR_INVALID: return "invalid argument";
    case IB_ERR_CUDA: return "CUDA error";
    case IB_ERR_NONFINITE: return "infinite flux";
    case IB_ERR_BODY_OUT_OF_GRID: return "body outside the finest grid";
    case IB_ERR_SINGULAR: return "singular Schur matrix";
    case IB_ERR_CG_MAXITER: return "Schur CG iteration cap reached";
    case IB_ERR_UNSUPPORTED: return "unsupported";
    case IB_ERR_TIMEOUT: return "device pipeline wait timed out";
    default: return "unknown status";
  }
}

const char* ib_last_error(const ib_handle* h) {
  if (h) return h->err.c_str();
  std::lock_guard<std::mutex> lock(g_err_mu);
  return g_create_err.c_str();
}

int ib_create(const ib_problem* p, ib_handle** out) {
  ib::Range nvtx_range("ib_create");
  const auto t_start = std::chrono::steady_clock::now();
  ib_handle* h = nullptr;
  if (!p || !out) return fail(nullptr, IB_ERR_INVALID, "null argument");
  *out = nullptr;
  if (p->nlevels < 1 || p->nx < 8 || p->ny < 8 || !(p->h > 0) || !(p->dt > 0) || !(p->re > 0))
    return fail(nullptr, IB_ERR_INVALID, "invalid grid or scheme parameters");
  if (!dst_axis_supported(p->nx) || !dst_axis_supported(p->ny))
    return fail(nullptr, IB_ERR_INVALID,
                "nx and ny must be multiples of 4, at most 2048, with n/2 a product of 2, 3 and 5");
  if (p->precision != IB_PREC_FP64 && p->precision != IB_PREC_MIXED && p->precision != IB_PREC_MIXED_TC)
    return fail(nullptr, IB_ERR_UNSUPPORTED, "precision mode not available");
  if (p->motion != IB_MOTION_STATIC && p->motion != IB_MOTION_PRESCRIBED)
    return fail(nullptr, IB_ERR_INVALID, "unknown body motion");
  int nb = 0;
  if (p->nbodies < 0) return fail(nullptr, IB_ERR_INVALID, "negative body count");
  for (int b = 0; b < p->nbodies; ++b) {
    if (!p->body_npoints || p->body_npoints[b] < 0) return fail(nullptr, IB_ERR_INVALID, "bad body point count");
    nb += p->body_npoints[b];
  }
  if (nb > 0 && (!p->xb || !p->ds)) return fail(nullptr, IB_ERR_INVALID, "missing body points");
  DeviceGuard dev_guard_(p->device);
  h = new ib_handle();
  h->device = p->device;
  cudaError_t e = dev_guard_.err;
  if (e != cudaSuccess) { int rc = fail(nullptr, IB_ERR_CUDA, "cudaSetDevice", e); delete h; return rc; }
  e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) { int rc = fail(nullptr, IB_ERR_CUDA, "cudaStreamCreate", e); h->stream = nullptr; destroy_handle(h); return rc; }
  auto bail = [&](int rc) {
    {
      std::lock_guard<std::mutex> lock(g_err_mu);
      g_create_err = h->err;
    }
    destroy_handle(h);
    return rc;
  };
  h->g = make_geometry(p->nx, p->ny, p->nlevels, p->h, p->x0, p->y0);
  if ((e = cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking)) != cudaSuccess) {
    h->side = nullptr;
    return bail(fail(h, IB_ERR_CUDA, "cudaStreamCreate", e));
  }
  h->fork_ev.assign(p->nlevels + 1, nullptr);
  for (auto& ev : h->fork_ev)
    if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
      ev = nullptr;
      return bail(fail(h, IB_ERR_CUDA, "cudaEventCreate", e));
    }
  h->dt = p->dt;
  h->re = p->re;
  h->beta0 = p->beta0;
  h->beta1 = p->beta1;
  h->nbodies = p->nbodies;
  h->nb = nb;
  h->nf = 2 * nb;
  if (p->scheme != IB_SCHEME_CNAB && p->scheme != IB_SCHEME_RKC) return bail(fail(h, IB_ERR_INVALID, "unknown scheme"));
  h->scheme = p->scheme;
  if (h->scheme == IB_SCHEME_RKC) {
    if (p->precision != IB_PREC_FP64)
      return bail(fail(h, IB_ERR_UNSUPPORTED, "the Runge-Kutta-Chebyshev scheme is FP64 only"));
    if (p->motion != IB_MOTION_STATIC)
      return bail(fail(h, IB_ERR_UNSUPPORTED, "the Runge-Kutta-Chebyshev scheme takes bodies fixed in the grid"));
    if (p->rkc_stages < 0 || p->rkc_stages == 1 || p->rkc_stages > 64)
      return bail(fail(h, IB_ERR_INVALID, "rkc_stages must be 0 (automatic) or 2..64"));
    // the fewest stages whose stability interval covers 1.5 x dt x the finest level's viscous
    // spectral radius 8 / (Re h^2)
    const double need = 1.5 * p->dt * 8.0 / (p->re * p->h * p->h);
    int S = p->rkc_stages;
    if (S == 0) {
      S = 2;
      while (S < 64 && rkc_coefficients(S, h->rkc_mu, h->rkc_nu, h->rkc_mut, h->rkc_gamt) < need) ++S;
    }
    rkc_coefficients(S, h->rkc_mu, h->rkc_nu, h->rkc_mut, h->rkc_gamt);
    h->rkc_s = S;
  }
  // IB_PREC_MIXED_TC is the mixed-precision solve with the tensor-core transform passes
  h->precision = p->precision == IB_PREC_FP64 ? IB_PREC_FP64 : IB_PREC_MIXED;
  const bool want_tc = p->precision == IB_PREC_MIXED_TC;
  if (want_tc && !(sgemm_axis_supported(p->nx) && sgemm_axis_supported(p->ny)))
    return bail(fail(h, IB_ERR_UNSUPPORTED, "tensor-core transforms need both axes a multiple of 128 cells"));
  h->motion = p->motion;
  h->hist_cap = p->history_capacity > 0 ? p->history_capacity : 4096;
  if (p->refine_sweeps < 0 || p->refine_sweeps > 2) return bail(fail(h, IB_ERR_INVALID, "refine_sweeps must be 0, 1 or 2"));
  h->refine = p->refine_sweeps == 1 ? 1 : 2;
  h->refine_coarse = p->refine_sweeps == 0 ? 1 : h->refine;
  h->coarse_from = 2;
  if (const char* env = std::getenv("IBGB300_REFINE_COARSE")) {
    const int v = std::atoi(env);
    if (v >= 1 && v <= 2) h->refine_coarse = v;
  }
  if (const char* env = std::getenv("IBGB300_COARSE_FROM")) {
    const int v = std::atoi(env);
    if (v >= 1) h->coarse_from = v;
  }
  if (const char* env = std::getenv("IBGB300_NO_GRAPH")) h->use_graph = !(env[0] == '1');
  if (const char* env = std::getenv("IBGB300_PDL")) h->use_pdl = env[0] == '1';
  // mixed precision with two sweeps: the trial Crank-Nicolson solve starts from Gamma_n (two
  // FP32 transform solves instead of three; IBGB300_CN_PREDICTOR=0 keeps three)
  h->cn_pred = h->refine >= 2;
  if (const char* env = std::getenv("IBGB300_CN_PREDICTOR")) h->cn_pred = h->cn_pred && env[0] != '0';
  if (const char* env = std::getenv("IBGB300_PC_ASSEMBLY")) h->asm_fp64 = std::strcmp(env, "fp64") == 0;
  // FP32 (mixed) transforms run faster one warp per line where both axes allow it
  // (IBGB300_DST=warp|stockham overrides the choice); FP64 ones have one form (dstfx.cu)
  const bool wsup = wdst_axis_supported(p->nx) && wdst_axis_supported(p->ny);
  h->wdst = wsup && p->precision != IB_PREC_FP64;
  h->gdst = want_tc;
  bool pin_form = want_tc, pin_v2f = false;
  if (const char* env = std::getenv("IBGB300_DST")) {
    if (std::strcmp(env, "stockham") == 0) { h->wdst = false; pin_form = true; }
    if (std::strcmp(env, "warp") == 0) { h->wdst = wsup; pin_form = true; }
  }
  // Mixed handles solve in fixed point too, float-float in and out, unless the FP32 passes are asked for
  // (one sweep, IBGB300_DST, IB_PREC_MIXED_TC): one such solve costs 1.1 FP32 transform solves at 256^2
  // and two at 1024^2, where two to three FP32 solves made a refined one.  Steps, against FP32 in its
  // better order: 256 x 192 x 3 247 -> 187 us, 1024^2 x 4 1114 -> 898, 2048^2 x 5 4372 -> 3932.
  h->fx_solve = h->precision == IB_PREC_MIXED && h->refine >= 2 && !pin_form;
  // the setup-time autotuner (autotune() above) replaces these size rules unless switched off
  const char* tune_env = std::getenv("IBGB300_AUTOTUNE");
  const bool autotune_on = !(tune_env && tune_env[0] == '0');
  const Geometry& g = h->g;
  const int L = g.nlev;
  const int64_t nG = g.nG;
  if ((e = h->axx.build(g.nx)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "x transform tables", e));
  if ((e = h->axy.build(g.ny)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "y transform tables", e));
  if (h->precision == IB_PREC_MIXED) {
    if ((e = h->axx32.build(g.nx)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "x transform tables", e));
    if ((e = h->axy32.build(g.ny)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "y transform tables", e));
  }
  if (h->gdst) {
    if ((e = h->sgx.build(g.nx)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "x sine-matrix image", e));
    if ((e = h->sgy.build(g.ny)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "y sine-matrix image", e));
  }
#define AL(ptr, n)                                                                       \
  do {                                                                                   \
    cudaError_t ea = h->alloc(&(ptr), (size_t)(n));                                      \
    if (ea != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "device allocation", ea));   \
  } while (0)
  AL(h->G[0], L * nG); AL(h->G[1], L * nG);
  AL(h->N[0], L * nG); AL(h->N[1], L * nG);
  AL(h->psi, L * nG); AL(h->q, (int64_t)L * g.nq);
  AL(h->fb, h->nf);
  AL(h->rhs, L * nG); AL(h->w1, L * nG); AL(h->w2, L * nG);
  AL(h->qs1, g.nq); AL(h->qtmp, g.nq); AL(h->gtmp, nG);
  AL(h->bcn, (int64_t)L * g.nbc); AL(h->edges, (int64_t)L * (2 * (g.nx - 1) + 2 * (g.ny - 1)));
  AL(h->rings, (int64_t)L * g.nbc);
  AL(h->mLap, nG); AL(h->mCN1, L * nG); AL(h->mCN2, L * nG);
  AL(h->d_fac, L); AL(h->d_q0, 2 * L); AL(h->d_inv_hc2, L); AL(h->d_alpha, L);
  AL(h->d_one, L); AL(h->d_zero, 1);
  if (h->precision == IB_PREC_MIXED) {
    AL(h->mLap32, nG); AL(h->mCN1_32, L * nG);
    AL(h->w32, L * nG); AL(h->x032, L * nG);
    if (h->gdst) AL(h->gw32, L * nG);
    if (h->refine >= 2) { AL(h->x132, L * nG); AL(h->r1, L * nG); }
    AL(h->conv, (int64_t)L * (g.nq > nG ? g.nq : nG));
    // Vort2Flux over all levels at once: two refinement sweeps, one-warp line passes on both
    // axes.  By measurement on GB300 (mixed step, device time) it is the faster order while one
    // level's passes leave the GPU part idle: 0.32 vs 0.41 ms at 256^2 x 3 levels, 0.64 vs 0.80
    // at 512^2 x 4, 1.41 vs 1.47 at 1024^2 x 4 (and C_L/C_D 2e-10 from FP64 instead of 2e-8),
    // but 6.15 vs 5.84 at 2048^2 x 5; so up to 2^20 cells per level.  IBGB300_V2F=levels|
    // sequential overrides the choice.
    const bool lv_base = wsup && L > 1 && h->refine >= 2 && h->axx32.d.wNL == 32 && h->axy32.d.wNL == 32;
    const bool lv_ok = lv_base && h->wdst && !h->gdst;
    h->v2f_ok = lv_ok;
    h->v2f_auto = lv_ok && (int64_t)g.nx * g.ny <= (int64_t(1) << 20);
    h->v2f_levels = h->v2f_auto;
    if (const char* env = std::getenv("IBGB300_V2F")) {
      if (std::strcmp(env, "sequential") == 0) { h->v2f_levels = false; pin_v2f = true; }
      if (std::strcmp(env, "levels") == 0) { h->v2f_levels = lv_ok; pin_v2f = true; }
    }
  }
  AL(h->d_counter, 1); AL(h->d_box, 4);
  if (h->scheme == IB_SCHEME_RKC) {
    AL(h->rkY[0], L * nG); AL(h->rkY[1], L * nG); AL(h->rkF0, L * nG);
    AL(h->d_alpha_rkc, L); AL(h->d_fac_rkc, L);
  }
  if (h->precision == IB_PREC_MIXED && h->cn_pred && !h->fx_solve) AL(h->cprev, nG);
  for (auto& ev : h->stress_ev)
    if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
      ev = nullptr;
      return bail(fail(h, IB_ERR_CUDA, "cudaEventCreate", e));
    }
  AL(h->cdcl, 2 * (h->nbodies > 0 ? h->nbodies : 1));
  AL(h->hist, (int64_t)h->hist_cap * 2 * (h->nbodies > 0 ? h->nbodies : 1));
  AL(h->stress, h->nf);
  {
    const size_t n = sizeof(double) * (2 * (h->nbodies > 0 ? h->nbodies : 1) + h->nf);
    if ((e = cudaMallocHost(&h->status, 4 * sizeof(int))) != cudaSuccess) {
      h->status = nullptr;
      return bail(fail(h, IB_ERR_CUDA, "pinned status", e));
    }
    std::memset(h->status, 0, 4 * sizeof(int));
    if ((e = cudaMallocHost(&h->h_stress, n)) != cudaSuccess) {
      h->h_stress = nullptr;
      return bail(fail(h, IB_ERR_CUDA, "pinned stress", e));
    }
    std::memset(h->h_stress, 0, n);
  }
  if ((e = cudaMallocHost(&h->h_q0, sizeof(double) * kQ0Slots * (2 * L + 6 * (h->nbodies + 1)))) != cudaSuccess) {
    h->h_q0 = nullptr;
    return bail(fail(h, IB_ERR_CUDA, "pinned staging", e));
  }
  // The copies of the set-up go through the legacy stream, which h->stream neither waits for nor holds up: they
  // begin when the arrays are zeroed and have landed before anything reads them.
  auto copies_begin = [&] { return cudaStreamSynchronize(h->stream); };
  auto copies_end = [&] { return cudaStreamSynchronize(nullptr); };
  {
    std::vector<double> lap, cn1, cn2;
    build_multipliers(h, lap, cn1, cn2);
    if ((e = copies_begin()) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
    std::vector<double> fac(L), ihc(L), alpha(L);
    for (int l = 0; l < L; ++l) {
      const double hc = g.h * std::ldexp(1.0, l);
      fac[l] = 0.25 * h->dt / (h->re * (hc * hc));    // timestepping.jl:50
      ihc[l] = 1.0 / (hc * hc);                       // cnab/ops.jl:162-163
      alpha[l] = h->dt / (2.0 * h->re * (hc * hc));   // cnab/ops.jl:26
    }
    if ((e = cudaMemcpy(h->mLap, lap.data(), sizeof(double) * lap.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->mCN1, cn1.data(), sizeof(double) * cn1.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->mCN2, cn2.data(), sizeof(double) * cn2.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->d_fac, fac.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->d_inv_hc2, ihc.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->d_alpha, alpha.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
    std::vector<double> ones(L, 1.0);
    if ((e = cudaMemcpy(h->d_one, ones.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
    if (h->scheme == IB_SCHEME_RKC) {
      // explicit viscous term nu lap / hc^2 and its ring weight, per level
      std::vector<double> visc(L);
      for (int l = 0; l < L; ++l) {
        const double hc = g.h * std::ldexp(1.0, l);
        visc[l] = 1.0 / (h->re * hc * hc);
      }
      if ((e = cudaMemcpy(h->d_alpha_rkc, visc.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess ||
          (e = cudaMemcpy(h->d_fac_rkc, visc.data(), sizeof(double) * L, cudaMemcpyHostToDevice)) != cudaSuccess)
        return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
    }
    if (h->precision == IB_PREC_MIXED) {
      std::vector<float> l32(lap.begin(), lap.end()), c32(cn1.begin(), cn1.end());
      if ((e = cudaMemcpy(h->mLap32, l32.data(), sizeof(float) * l32.size(), cudaMemcpyHostToDevice)) != cudaSuccess ||
          (e = cudaMemcpy(h->mCN1_32, c32.data(), sizeof(float) * c32.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
        return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
    }
    if ((e = copies_end()) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "parameter upload", e));
  }
  {
    const bool mixed = h->precision == IB_PREC_MIXED;
    const bool lv_base = mixed && wsup && L > 1 && h->refine >= 2 && h->axx32.d.wNL == 32 && h->axy32.d.wNL == 32;
    // mixed precision only: the FP64 path keeps its fixed, measured kernel rule, so that its
    // results are the same bits from run to run
    const bool tune_form = mixed && autotune_on && !pin_form;
    const bool tune_v2f = mixed && autotune_on && !pin_v2f && lv_base;
    if (tune_form || tune_v2f) {
      int rc = autotune(h, tune_form, tune_v2f, lv_base);
      if (rc != IB_OK) return bail(rc);
    } else if (mixed && h->v2f_levels && !h->rplan.St && (e = h->rplan.build(g, h->mLap)) != cudaSuccess) {
      return bail(fail(h, IB_ERR_CUDA, "ring transfer tables", e));
    }
    if (mixed) {
      h->v2f_ok = lv_base && h->wdst && !h->gdst;
      if (h->tuned) h->v2f_auto = h->v2f_levels;
      else h->v2f_auto = h->v2f_auto && h->v2f_ok;
    }
    if (!mixed || h->fx_solve) {
      // fixed-point Vort2Flux
      h->tuned_levels = h->v2f_levels;
      h->v2f_fx = true;
      // by measurement (steps, all levels at once / level by level, us): 128^2 x 2 125 / 125, x 3 148 /
      // 162; 256^2 x 3 196 / 209, x 4 205 / 258; 384 x 256 x 3 224 / 235; 512^2 x 3 344 / 332, x 4 404 /
      // 422; 1024^2 x 3 837 / 819, x 4 997 / 1032; 2048^2 x 5 4442 / 4633
      // Long, narrow grids keep all modes of their long sides, and the rings' sums outweigh the passes saved
      // (Vort2Flux calls, all levels / level by level, us, and sums in 2^20: 256 x 32 x 4 99 / 122, 0.9; 512 x
      // 64 x 4 127 / 137, 3.4; 1024 x 128 x 4 169 / 170, 7.0; 1024 x 64 x 4 204 / 168, 12.8; 2048 x 256 x 4
      // 291 / 221, 12.0; 1200 x 12 x 4 227 / 160, 16.7).  Large square ones have as many, beside longer passes
      // (2048^2 x 5: 9.6)
      const int64_t cells = (int64_t)g.nx * g.ny;
      h->v2f_auto = (L >= 4 || (L == 3 && cells <= (int64_t(1) << 17))) &&
                    v2f_ring_work(g) <= std::max<int64_t>(int64_t(1) << 22, 4 * cells);
      // a mixed handle takes the order on request where its grid has one-warp lines, whatever FP32 passes the tuner
      // chose (else the rule's order stands)
      if (mixed) h->v2f_ok = lv_base;
      h->v2f_levels = h->v2f_auto;
      if (const char* env = std::getenv("IBGB300_V2F")) {
        // as ib_set_vort2flux_order: the reference's order of a mixed handle is that of the FP32 transforms
        if (std::strcmp(env, "sequential") == 0) h->v2f_levels = false, h->v2f_fx = !mixed;
        if (std::strcmp(env, "levels") == 0) h->v2f_levels = mixed ? h->v2f_ok || h->v2f_auto : L > 1;
      }
      if (!mixed) h->v2f_auto = h->v2f_levels;
      if (h->v2f_levels && ((!h->rplan.St && (e = h->rplan.build(g, h->mLap)) != cudaSuccess) ||
                            (e = h->rplan.build_fx(g, h->stream)) != cudaSuccess))
        return bail(fail(h, IB_ERR_CUDA, "ring transfer tables", e));
    }
  }
  if (nb > 0) {
    const bool moving = h->motion == IB_MOTION_PRESCRIBED;
    AL(h->xb, 2 * nb); AL(h->ds, nb); AL(h->weight, (int64_t)nb * 2 * kWin2);
    AL(h->body_idx, 2 * nb); AL(h->body_start, h->nbodies + 1); AL(h->ftmp, h->nf);
    if (!moving) {
      AL(h->bmat, (int64_t)h->nf * h->nf); AL(h->binv_cm, (int64_t)h->nf * h->nf);
      AL(h->binv_rm, (int64_t)h->nf * h->nf);
    } else {
      AL(h->xb_body, 2 * nb); AL(h->vb, 2 * nb); AL(h->d_kin, 6 * h->nbodies); AL(h->body_of, nb);
      AL(h->cg_r, h->nf); AL(h->cg_p, h->nf); AL(h->cg_Ap, h->nf); AL(h->cg_sc, 8); AL(h->fb_prev, h->nf);
      AL(h->fb_last, h->nf); AL(h->cg_z, h->nf); AL(h->d_cgctl, 4); AL(h->d_cgout, 4);
      if ((e = cudaMallocHost(&h->h_mslot, sizeof(double) * kMaxStepsPerLaunch * (2 * L + 6 * h->nbodies))) !=
          cudaSuccess) {
        h->h_mslot = nullptr;
        return bail(fail(h, IB_ERR_CUDA, "pinned staging", e));
      }
      if ((e = cudaMallocHost(&h->h_cgout, sizeof(double) * 4 * kMaxStepsPerLaunch)) != cudaSuccess) {
        h->h_cgout = nullptr;
        return bail(fail(h, IB_ERR_CUDA, "pinned staging", e));
      }
      if ((e = cudaStreamCreateWithFlags(&h->loop_stream, cudaStreamNonBlocking)) != cudaSuccess) {
        h->loop_stream = nullptr;
        return bail(fail(h, IB_ERR_CUDA, "cudaStreamCreate", e));
      }
      AL(h->Gw, L * nG); AL(h->Pw, L * nG); AL(h->qw, g.nq); AL(h->rings_w, (int64_t)L * g.nbc);
      if ((e = cudaMallocHost(&h->h_sc, sizeof(double) * 8)) != cudaSuccess) {
        h->h_sc = nullptr;
        return bail(fail(h, IB_ERR_CUDA, "pinned CG scalars", e));
      }
    }
    std::vector<int> bs(h->nbodies + 1, 0), bof(nb);
    for (int b = 0; b < h->nbodies; ++b) {
      bs[b + 1] = bs[b] + p->body_npoints[b];
      for (int k = bs[b]; k < bs[b + 1]; ++k) bof[k] = b;
    }
    if ((e = copies_begin()) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "body upload", e));
    if ((e = cudaMemcpy(moving ? h->xb_body : h->xb, p->xb, sizeof(double) * 2 * nb, cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (e = cudaMemcpy(h->ds, p->ds, sizeof(double) * nb, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (e = cudaMemcpy(h->body_start, bs.data(), sizeof(int) * bs.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail(fail(h, IB_ERR_CUDA, "body upload", e));
    if (moving && (e = cudaMemcpy(h->body_of, bof.data(), sizeof(int) * nb, cudaMemcpyHostToDevice)) != cudaSuccess)
      return bail(fail(h, IB_ERR_CUDA, "body upload", e));
    if ((e = copies_end()) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "body upload", e));
    if (!moving) {
      if ((e = reg_update(g, h->xb, nb, h->body_idx, h->weight, h->status, h->stream)) != cudaSuccess)
        return bail(fail(h, IB_ERR_CUDA, "delta weights", e));
      if ((e = body_box(g, h->body_idx, nb, h->d_box, h->stream)) != cudaSuccess)
        return bail(fail(h, IB_ERR_CUDA, "body box", e));
      h->box_ready = true;
      int rc = check_status(h);
      if (rc != IB_OK) return bail(rc);
    }
  }
#undef AL
  {
    int rc = prime_kernels(h);
    if (rc != IB_OK) return bail(rc);
  }
  if (nb > 0 && h->motion == IB_MOTION_STATIC) {
    int rc = assemble_schur(h);
    if (rc != IB_OK) return bail(rc);
    rc = check_status(h);
    if (rc != IB_OK) return bail(rc);
  }
  if (h->motion == IB_MOTION_PRESCRIBED) {
    h->use_moving_graph = h->use_graph;  // IBGB300_NO_GRAPH=1 keeps every moving step eager
    h->use_graph = false;
  }
  if (h->use_graph) {
    int rc = capture_graphs(h);
    if (rc != IB_OK) return bail(rc);
  }
  if ((e = cudaStreamSynchronize(h->stream)) != cudaSuccess) return bail(fail(h, IB_ERR_CUDA, "setup", e));
  h->setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
  *out = h;
  return IB_OK;
}

int ib_destroy(ib_handle* h) {
  destroy_handle(h);
  return IB_OK;
}

int ib_set_state(ib_handle* h, const double* gamma, const double* q, const double* psi, const double* nonlin1,
                 const double* nonlin2, const double* fb, double t) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  const Geometry& g = h->g;
  const size_t nGL = sizeof(double) * g.nlev * g.nG, nqL = sizeof(double) * g.nlev * g.nq;
  const int p = h->parity;
  cudaStream_t s = h->stream;
  CK(cudaStreamSynchronize(s));
  if (gamma) CK(cudaMemcpyAsync(h->G[p], gamma, nGL, cudaMemcpyHostToDevice, s));
  if (q) CK(cudaMemcpyAsync(h->q, q, nqL, cudaMemcpyHostToDevice, s));
  if (psi) CK(cudaMemcpyAsync(h->psi, psi, nGL, cudaMemcpyHostToDevice, s));
  if (nonlin1) CK(cudaMemcpyAsync(h->N[p], nonlin1, nGL, cudaMemcpyHostToDevice, s));
  if (nonlin2) CK(cudaMemcpyAsync(h->N[p ^ 1], nonlin2, nGL, cudaMemcpyHostToDevice, s));
  if (fb && h->nf) CK(cudaMemcpyAsync(h->fb, fb, sizeof(double) * h->nf, cudaMemcpyHostToDevice, s));
  if (h->precision == IB_PREC_MIXED) {
    // the mixed mode keeps its state as float-float pairs: convert in place
    const int64_t nG = (int64_t)g.nlev * g.nG, nq = (int64_t)g.nlev * g.nq;
    if (gamma) k_to_df64<<<conv_blocks(nG), 256, 0, s>>>(h->G[p], nG);
    if (q) k_to_df64<<<conv_blocks(nq), 256, 0, s>>>(h->q, nq);
    if (psi) k_to_df64<<<conv_blocks(nG), 256, 0, s>>>(h->psi, nG);
    if (nonlin1) k_to_df64<<<conv_blocks(nG), 256, 0, s>>>(h->N[p], nG);
    if (nonlin2) k_to_df64<<<conv_blocks(nG), 256, 0, s>>>(h->N[p ^ 1], nG);
    CK(cudaGetLastError());
  }
  // the batched Vort2Flux predicts psi and the rings from the previous call: a new state starts
  // from its own psi (or zero) and zero rings
  // the projection's correction predicts the next one: a new state starts from zero
  if (h->cprev) CK(cudaMemsetAsync(h->cprev, 0, sizeof(double) * g.nG, s));
  if (h->precision == IB_PREC_MIXED && h->v2f_levels) {
    if (!psi) CK(cudaMemsetAsync(h->psi, 0, nGL, s));
    CK(cudaMemsetAsync(h->rings, 0, sizeof(double) * g.nlev * g.nbc, s));
    if (h->rings_w) CK(cudaMemsetAsync(h->rings_w, 0, sizeof(double) * g.nlev * g.nbc, s));
    if (h->Pw) CK(cudaMemsetAsync(h->Pw, 0, nGL, s));
  }
  CK(cudaStreamSynchronize(s));
  h->t = t;
  return IB_OK;
}

int ib_get_state(ib_handle* h, double* gamma, double* q, double* psi, double* nonlin1, double* nonlin2, double* fb,
                 double* t) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  const Geometry& g = h->g;
  const size_t nGL = sizeof(double) * g.nlev * g.nG, nqL = sizeof(double) * g.nlev * g.nq;
  const int p = h->parity;
  cudaStream_t s = h->stream;
  // mixed mode: each float-float array is widened into the conversion buffer, then copied
  auto pull = [&](double* dst, double* src, size_t bytes) -> cudaError_t {
    if (h->precision != IB_PREC_MIXED) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    const int64_t n = (int64_t)(bytes / sizeof(double));
    k_from_df64<<<conv_blocks(n), 256, 0, s>>>(view<df64>(src), h->conv, n);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(dst, h->conv, bytes, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(s);  // the buffer is reused by the next array
  };
  if (gamma) CK(pull(gamma, h->G[p], nGL));
  if (q) CK(pull(q, h->q, nqL));
  if (psi) CK(pull(psi, h->psi, nGL));
  if (nonlin1) CK(pull(nonlin1, h->N[p], nGL));
  if (nonlin2) CK(pull(nonlin2, h->N[p ^ 1], nGL));
  if (fb && h->nf) CK(cudaMemcpyAsync(fb, h->fb, sizeof(double) * h->nf, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (t) *t = h->t;
  return check_status(h);
}

// ---- checkpoint files ------------------------------------------------------------------------
// Layout (little-endian): 8-byte magic "IBGB300C", int32 version (1), int32 nx, ny, nlevels,
// npoints, moving (1 if the F_{n-2} block follows), two int32 zeros, double t, int64 steps, then
// FP64 arrays in the ABI's column-major layouts: Gamma, q, psi, nonlin[1], nonlin[2]
// (nlevels x (nx-1)(ny-1) or nlevels x nq each), Fb (2 npoints) and, for moving bodies, the
// previous step's Fb (the CG warm start's history).
namespace {
constexpr char kCkptMagic[8] = {'I', 'B', 'G', 'B', '3', '0', '0', 'C'};
struct CkptHeader {
  char magic[8];
  int32_t version, nx, ny, nlevels, npoints, moving, reserved0, reserved1;
  double t;
  int64_t steps;
};
static_assert(sizeof(CkptHeader) == 56, "checkpoint header layout");
}  // namespace

int ib_checkpoint_save(ib_handle* h, const char* path) {
  ib::Range nvtx_range("ib_checkpoint_save");
  if (!h || !path) return IB_ERR_INVALID;
  const Geometry& g = h->g;
  const size_t nGL = (size_t)g.nlev * g.nG, nqL = (size_t)g.nlev * g.nq;
  std::vector<double> buf(4 * nGL + nqL + 2 * (size_t)h->nf);
  double* gam = buf.data();
  double* q = gam + nGL;
  double* psi = q + nqL;
  double* n1 = psi + nGL;
  double* n2 = n1 + nGL;
  double* fb = n2 + nGL;
  double t = 0.0;
  int rc = ib_get_state(h, gam, q, psi, n1, n2, fb, &t);
  if (rc != IB_OK) return rc;
  const bool moving = h->motion == IB_MOTION_PRESCRIBED && h->nf > 0;
  if (moving) {
    DeviceGuard dev_guard_(h->device);
    CK(dev_guard_.err);
    CK(cudaMemcpy(fb + h->nf, h->fb_prev, sizeof(double) * h->nf, cudaMemcpyDeviceToHost));
  }
  CkptHeader hd{};
  std::memcpy(hd.magic, kCkptMagic, 8);
  hd.version = 1;
  hd.nx = g.nx; hd.ny = g.ny; hd.nlevels = g.nlev; hd.npoints = h->nb; hd.moving = moving ? 1 : 0;
  hd.t = t;
  hd.steps = h->steps;
  FILE* f = std::fopen(path, "wb");
  if (!f) return fail(h, IB_ERR_INVALID, "checkpoint: cannot open the file for writing");
  const size_t nvals = 4 * nGL + nqL + (size_t)h->nf * (moving ? 2 : 1);
  const bool ok = std::fwrite(&hd, sizeof(hd), 1, f) == 1 && std::fwrite(buf.data(), sizeof(double), nvals, f) == nvals;
  const bool closed = std::fclose(f) == 0;
  if (!ok || !closed) return fail(h, IB_ERR_INVALID, "checkpoint: write failed");
  return IB_OK;
}

int ib_checkpoint_load(ib_handle* h, const char* path) {
  ib::Range nvtx_range("ib_checkpoint_load");
  if (!h || !path) return IB_ERR_INVALID;
  const Geometry& g = h->g;
  FILE* f = std::fopen(path, "rb");
  if (!f) return fail(h, IB_ERR_INVALID, "checkpoint: cannot open the file");
  CkptHeader hd{};
  if (std::fread(&hd, sizeof(hd), 1, f) != 1 || std::memcmp(hd.magic, kCkptMagic, 8) != 0 || hd.version != 1) {
    std::fclose(f);
    return fail(h, IB_ERR_INVALID, "checkpoint: not a version-1 libibgb300 checkpoint");
  }
  const bool moving = h->motion == IB_MOTION_PRESCRIBED && h->nf > 0;
  if (hd.nx != g.nx || hd.ny != g.ny || hd.nlevels != g.nlev || hd.npoints != h->nb || (hd.moving != 0) != moving) {
    std::fclose(f);
    return fail(h, IB_ERR_INVALID, "checkpoint: grid, levels, points or body motion differ from the handle's");
  }
  const size_t nGL = (size_t)g.nlev * g.nG, nqL = (size_t)g.nlev * g.nq;
  const size_t nvals = 4 * nGL + nqL + (size_t)h->nf * (moving ? 2 : 1);
  std::vector<double> buf(nvals);
  const bool ok = std::fread(buf.data(), sizeof(double), nvals, f) == nvals;
  std::fclose(f);
  if (!ok) return fail(h, IB_ERR_INVALID, "checkpoint: file is shorter than its header says");
  double* gam = buf.data();
  double* q = gam + nGL;
  double* psi = q + nqL;
  double* n1 = psi + nGL;
  double* n2 = n1 + nGL;
  double* fb = n2 + nGL;
  int rc = ib_set_state(h, gam, q, psi, n1, n2, h->nf ? fb : nullptr, hd.t);
  if (rc != IB_OK) return rc;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  if (moving) {
    CK(cudaMemcpy(h->fb_prev, fb + h->nf, sizeof(double) * h->nf, cudaMemcpyHostToDevice));
    for (auto& ge : h->mgexec)
      if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
  }
  h->steps = hd.steps;
  // the C_D / C_L history continues at the restored step (its earlier entries are not in the
  // file)
  const int counter = (int)(hd.steps % h->hist_cap);
  CK(cudaMemcpy(h->d_counter, &counter, sizeof(int), cudaMemcpyHostToDevice));
  return IB_OK;
}

int ib_advance(ib_handle* h, double t, double u, double v) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  int rc = one_step(h, t, u, v);
  if (rc != IB_OK) return rc;
  return check_status(h);
}

int ib_advance_n(ib_handle* h, int32_t n, const double* t, const double* uv) {
  ib::Range nvtx_range("ib_advance_n");
  if (!h || n < 0 || (n > 0 && (!t || !uv))) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  for (int i = 0; i < n; ++i) {
    int rc = one_step(h, t[i], uv[2 * i], uv[2 * i + 1]);
    if (rc != IB_OK) return rc;
  }
  return check_status(h);
}

int ib_advance_kin(ib_handle* h, double t, double u, double v, const double* kin) {
  if (!h) return IB_ERR_INVALID;
  if (h->motion != IB_MOTION_PRESCRIBED) {
    if (kin) return fail(h, IB_ERR_INVALID, "kinematics given for bodies fixed in the grid");
    return ib_advance(h, t, u, v);
  }
  if (!kin) return fail(h, IB_ERR_INVALID, "moving bodies need kinematics");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  return moving_step_mode(h, t, u, v, kin);
}

int ib_advance_n_kin(ib_handle* h, int32_t n, const double* t, const double* uv, const double* kin) {
  ib::Range nvtx_range("ib_advance_n_kin");
  if (!h || n < 0 || (n > 0 && (!t || !uv))) return IB_ERR_INVALID;
  if (h->motion != IB_MOTION_PRESCRIBED) return ib_advance_n(h, n, t, uv);
  if (n > 0 && !kin) return fail(h, IB_ERR_INVALID, "moving bodies need kinematics");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  for (int i = 0; i < n; ++i) {
    int rc = moving_step_mode(h, t[i], uv[2 * i], uv[2 * i + 1], kin + (size_t)i * 6 * h->nbodies);
    if (rc != IB_OK) return rc;
  }
  return IB_OK;
}

int ib_set_cg_options(ib_handle* h, double tol, int32_t maxiter, int32_t warm_start) {
  if (!h || !(tol > 0) || maxiter < 1 || warm_start < IB_WARM_PREVIOUS || warm_start > IB_WARM_LEARNED)
    return IB_ERR_INVALID;
  h->cg_tol = tol;
  h->cg_maxiter = maxiter;
  h->warm_start = warm_start;
  return IB_OK;
}

int ib_set_cg_preconditioner(ib_handle* h, int32_t mode, int32_t refresh_steps) {
  if (!h || (mode != IB_PC_NONE && mode != IB_PC_SCHUR_REF) || refresh_steps < 0) return IB_ERR_INVALID;
  if (mode != IB_PC_NONE && h->motion != IB_MOTION_PRESCRIBED)
    return fail(h, IB_ERR_INVALID, "a CG preconditioner applies to moving bodies only");
  h->precond = mode;
  h->pc_refresh = refresh_steps;
  h->pc_step = -1;
  h->pc_base_iters = -1;
  return IB_OK;
}

int ib_set_vort2flux_order(ib_handle* h, int32_t order) {
  if (!h || order < IB_V2F_AUTO || order > IB_V2F_SEQUENTIAL) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  const bool mixed = h->precision == IB_PREC_MIXED;
  if (mixed && order == IB_V2F_LEVELS && !h->v2f_ok)
    return fail(h, IB_ERR_UNSUPPORTED, "the all-levels Vort2Flux needs one-warp line passes on both axes");
  const bool lv = (order == IB_V2F_LEVELS && h->g.nlev > 1) || (order == IB_V2F_AUTO && h->v2f_auto);
  const bool fx = !mixed || (h->fx_solve && order != IB_V2F_SEQUENTIAL);
  if (lv == h->v2f_levels && fx == h->v2f_fx) return IB_OK;
  CK(cudaStreamSynchronize(h->stream));
  if (lv) {
    cudaError_t e = cudaSuccess;
    if (!h->rplan.St && (e = h->rplan.build(h->g, h->mLap)) != cudaSuccess) h->rplan.release();
    if (e == cudaSuccess && fx) e = h->rplan.build_fx(h->g, h->stream);
    if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "ring transfer tables", e);
  }
  h->v2f_levels = lv;
  h->v2f_fx = fx;
  // the rings buffers then hold the other order's values: a predictor only, either is valid
  if (h->gexec[0]) {
    int rc = capture_graphs(h);
    if (rc != IB_OK) return rc;
  }
  for (auto& ge : h->mgexec)
    if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
  return IB_OK;
}

int ib_get_cg_preconditioner_stats(ib_handle* h, int32_t* assemblies, int64_t* last_step, double* last_seconds) {
  if (!h) return IB_ERR_INVALID;
  if (assemblies) *assemblies = h->pc_assemblies;
  if (last_step) *last_step = h->pc_step;
  if (last_seconds) *last_seconds = h->pc_assembly_s;
  return IB_OK;
}

int ib_get_cg_stats(ib_handle* h, int32_t count, int32_t* iterations, double* residuals) {
  if (!h || count < 0 || count > (int32_t)h->cg_iters.size()) return IB_ERR_INVALID;
  const size_t off = h->cg_iters.size() - (size_t)count;
  for (int i = 0; i < count; ++i) {
    if (iterations) iterations[i] = h->cg_iters[off + i];
    if (residuals) residuals[i] = h->cg_res[off + i];
  }
  return IB_OK;
}

int ib_get_body_points(ib_handle* h, double* xb, double* vb) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  if (h->nb == 0) return IB_OK;
  if (xb) CK(cudaMemcpyAsync(xb, h->xb, sizeof(double) * 2 * h->nb, cudaMemcpyDeviceToHost, h->stream));
  if (vb) {
    if (h->vb) CK(cudaMemcpyAsync(vb, h->vb, sizeof(double) * 2 * h->nb, cudaMemcpyDeviceToHost, h->stream));
    else std::memset(vb, 0, sizeof(double) * 2 * h->nb);
  }
  CK(cudaStreamSynchronize(h->stream));
  return IB_OK;
}

int ib_vort2flux(ib_handle* h) {
  ib::Range nvtx_range("ib_vort2flux");
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  if (h->precision == IB_PREC_MIXED)
    CK(vort2flux<df64>(h, view<df64>(h->G[h->parity]), view<df64>(h->psi), view<df64>(h->q), nullptr,
                       view<df64>(h->rings)));
  else
    CK(vort2flux<double>(h, h->G[h->parity], h->psi, h->q, nullptr, h->rings));
  CK(cudaStreamSynchronize(h->stream));
  return IB_OK;
}

int ib_get_stress(ib_handle* h, double* cd, double* cl, double* fb_surface) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  const int nbd = h->nbodies;
  if (nbd == 0) return IB_OK;
  CK(cudaStreamSynchronize(h->stream));
  const double* v = h->h_stress;
  if (fb_surface && h->nf) std::memcpy(fb_surface, v + 2 * nbd, sizeof(double) * h->nf);
  for (int b = 0; b < nbd; ++b) {
    if (cd) cd[b] = v[2 * b];
    if (cl) cl[b] = v[2 * b + 1];
  }
  return IB_OK;
}

int ib_get_force_history(ib_handle* h, int32_t count, double* cd, double* cl) {
  if (!h || count < 0) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  const int nbd = h->nbodies;
  if (nbd == 0 || count == 0) return IB_OK;
  if (count > h->hist_cap || count > h->steps) return fail(h, IB_ERR_INVALID, "history count exceeds recorded steps");
  std::vector<double> all((size_t)h->hist_cap * 2 * nbd);
  CK(cudaMemcpyAsync(all.data(), h->hist, sizeof(double) * all.size(), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int i = 0; i < count; ++i) {
    const int64_t step = h->steps - count + i;
    const int64_t slot = step % h->hist_cap;
    for (int b = 0; b < nbd; ++b) {
      if (cd) cd[(int64_t)i * nbd + b] = all[(size_t)slot * 2 * nbd + 2 * b];
      if (cl) cl[(int64_t)i * nbd + b] = all[(size_t)slot * 2 * nbd + 2 * b + 1];
    }
  }
  return IB_OK;
}

int64_t ib_step_count(const ib_handle* h) { return h ? h->steps : 0; }

int ib_synchronize(ib_handle* h) {
  if (!h) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  CK(cudaStreamSynchronize(h->stream));
  return check_status(h);
}

// ------------------------------------------------------------------------------------------------
// diagnostics (include/ibgb300_diag.h)
// ------------------------------------------------------------------------------------------------
int ib_get_info(ib_handle* h, ib_info* info) {
  if (!h || !info) return IB_ERR_INVALID;
  info->kernels_per_step = h->kernels_per_step;
  info->nx = h->g.nx;
  info->ny = h->g.ny;
  info->nlevels = h->g.nlev;
  info->nbodies = h->nbodies;
  info->npoints = h->nb;
  {
    std::lock_guard<std::mutex> lock(h->op_mu);
    info->device_bytes = h->device_bytes + h->rplan.bytes + (int64_t)sizeof(double) * h->op_cap;
  }
  info->setup_ms = h->setup_ms;
  info->vort2flux_order = h->v2f_levels ? IB_V2F_LEVELS : IB_V2F_SEQUENTIAL;
  info->transform_form = h->precision == IB_PREC_FP64 ? IB_FORM_FIXED
                         : h->gdst ? IB_FORM_TENSOR : (h->wdst ? IB_FORM_WARP : IB_FORM_STOCKHAM);
  info->scheme = h->scheme;
  info->rkc_stages = h->rkc_s;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device) != cudaSuccess) sms = 0;
  info->sm_count = sms;
  return IB_OK;
}

int ib_get_autotune(ib_handle* h, double* ms, int32_t* chosen) {
  if (!h) return IB_ERR_INVALID;
  if (ms)
    for (int i = 0; i < 12; ++i) ms[i] = h->tune_ms[i];
  if (chosen)
    *chosen = h->tuned ? ((h->gdst ? IB_FORM_TENSOR : (h->wdst ? IB_FORM_WARP : IB_FORM_STOCKHAM)) * 2 +
                          ((h->fx_solve ? h->tuned_levels : h->v2f_levels) ? 1 : 0)) * 2 + (h->axy32.d.wMinB == 8 ? 1 : 0)
                       : -1;
  return IB_OK;
}

int ib_advance_n_timed(ib_handle* h, int32_t n, const double* t, const double* uv, double* device_ms) {
  if (!h || n < 0 || (n > 0 && (!t || !uv))) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  CK(cudaEventRecord(e0, h->stream));
  int rc = IB_OK;
  for (int i = 0; i < n && rc == IB_OK; ++i) rc = one_step(h, t[i], uv[2 * i], uv[2 * i + 1]);
  CK(cudaEventRecord(e1, h->stream));
  CK(cudaEventSynchronize(e1));
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (device_ms) *device_ms = ms;
  if (rc != IB_OK) return rc;
  return check_status(h);
}

int ib_profile_steps(ib_handle* h, int32_t n, const double* t, const double* uv, int32_t kernel_class,
                     double* total_ms, int64_t* launches) {
  if (!h || n < 0 || (n > 0 && (!t || !uv)) || kernel_class < 0 || kernel_class >= kClassCount)
    return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  Prof prof;
  prof.cls = kernel_class;
  g_prof = &prof;
  const bool graph = h->use_graph;
  h->use_graph = false;
  int rc = IB_OK;
  for (int i = 0; i < n && rc == IB_OK; ++i) rc = one_step(h, t[i], uv[2 * i], uv[2 * i + 1]);
  h->use_graph = graph;
  g_prof = nullptr;
  cudaError_t e = cudaStreamSynchronize(h->stream);
  double sum = 0.0;
  for (size_t i = 0; i + 1 < prof.used; i += 2) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, prof.ev[i], prof.ev[i + 1]) == cudaSuccess) sum += ms;
  }
  for (auto ev : prof.ev) cudaEventDestroy(ev);
  if (total_ms) *total_ms = sum;
  if (launches) *launches = (int64_t)(prof.used / 2);
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "profiled steps", e);
  if (rc != IB_OK) return rc;
  return check_status(h);
}

// ------------------------------------------------------------------------------------------------
// operator entry points (device pointers)
// ------------------------------------------------------------------------------------------------
#define OP_BEGIN()                         \
  if (!h) return IB_ERR_INVALID;           \
  DeviceGuard dev_guard_(h->device);       \
  CK(dev_guard_.err);                      \
  const Geometry& g = h->g;                \
  cudaStream_t s = h->stream;              \
  (void)g;                                 \
  (void)s;
#define OP_END()                      \
  CK(cudaGetLastError());             \
  CK(cudaStreamSynchronize(s));       \
  return IB_OK;

}  // extern "C"

namespace {
// Work array of one operator call.  Up to the size of a step's work array it is the handle's own, kept
// from call to call (allocating and releasing it made a 64 x 48 Poisson call 34 us instead of 29) and locked
// until the call's kernels have finished, since calls from several threads may share a handle; larger
// ones are allocated for the call.
struct OpWork {
  ib_handle* h;
  std::unique_lock<std::mutex> lock;
  void* own = nullptr;

  explicit OpWork(ib_handle* handle) : h(handle), lock(handle->op_mu) {}
  cudaError_t get(double** p, int64_t n) {
    const int64_t most = std::max<int64_t>((int64_t)h->g.nlev * h->g.nG, (int64_t)h->g.nlev * h->g.nbc);
    if (n > most) {
      const cudaError_t e = cudaMalloc(&own, sizeof(double) * n);
      *p = static_cast<double*>(own);
      return e;
    }
    if (n > h->op_cap) {
      if (h->op_work) cudaFree(h->op_work);
      h->op_work = nullptr;
      h->op_cap = 0;
      const cudaError_t e = cudaMalloc(&h->op_work, sizeof(double) * n);
      if (e != cudaSuccess) return e;
      h->op_cap = n;
    }
    *p = h->op_work;
    return cudaSuccess;
  }
  void done() {
    cudaStreamSynchronize(h->stream);
    if (own) cudaFree(own);
    own = nullptr;
  }
};
}  // namespace

extern "C" {

int ib_op_dst2(ib_handle* h, int32_t batch, const double* in, double* out) {
  OP_BEGIN();
  if (batch < 1) return IB_ERR_INVALID;
  OpWork work(h);
  double* w;
  CK(work.get(&w, (int64_t)batch * g.nG));
  // RODFT00 in both dimensions = 4 F_y F_x (F: the half-scaled transform of dstfx.cu)
  cudaError_t e = fx_fwd<double>(g, h->axx.d, in, w, batch, nullptr, s);
  if (e == cudaSuccess) e = fx_ypass(g, h->axy.d, w, out, batch, nullptr, 0, 2, s);
  work.done();
  CK(e);
  OP_END();
}

int ib_op_sine_lines_tc(ib_handle* h, int32_t axis, int32_t rows, const float* in, float* out) {
  OP_BEGIN();
  if (rows < 1 || axis < 0 || axis > 1 || !in || !out) return IB_ERR_INVALID;
  const int n = axis == 0 ? g.nx : g.ny;
  if (!sgemm_axis_supported(n)) return fail(h, IB_ERR_UNSUPPORTED, "tensor-core transforms need a multiple of 128 cells");
  SineGemm& t = axis == 0 ? h->sgx : h->sgy;
  if (!t.img) CK(t.build(n));
  SgIn si{in, n - 1, rows, n - 1};
  SgOut so{};
  so.mode = 0; so.out = out; so.ld = n - 1; so.rpb = rows; so.ncols = n - 1;
  CK(sgemm_pass(t, si, so, h->status, s));
  CK(cudaStreamSynchronize(s));
  return check_status(h);
}

int ib_op_laplacian_inv(ib_handle* h, int32_t batch, const double* b, double* x) {
  OP_BEGIN();
  if (batch < 1) return IB_ERR_INVALID;
  OpWork work(h);
  double* w;
  CK(work.get(&w, (int64_t)batch * g.nG));
  cudaError_t e = poisson_fx<double>(h, b, x, batch, nullptr, op_lap(h), nullptr, w);
  work.done();
  CK(e);
  OP_END();
}

static int cn_op(ib_handle* h, int32_t lev, const double* b, double* x, bool inverse) {
  OP_BEGIN();
  if (lev < 1 || lev > g.nlev) return IB_ERR_INVALID;
  double *w, *m;
  CK(cudaMalloc(&w, sizeof(double) * g.nG));
  CK(cudaMalloc(&m, sizeof(double) * g.nG));
  cudaError_t e;
  const int64_t off = (int64_t)(lev - 1) * g.nG;
  if (inverse) {
    SolveOp op = op_cn1(h);
    op.m64 = h->mCN1 + off;
    e = poisson_fx<double>(h, b, x, 1, nullptr, op, nullptr, w);
  } else {
    // A multiplier = 16 * scale / Lambda_expl = 16 * scale * cn2 ; build it on the device
    e = cudaMemcpyAsync(m, h->mCN2 + off, sizeof(double) * g.nG, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = axpby<double>(m, m, 16.0 / (4.0 * g.nx * g.ny), 0.0, g.nG, s);
    SolveOp op = op_lap(h);
    op.m64 = m;
    if (e == cudaSuccess) e = poisson_fx<double>(h, b, x, 1, nullptr, op, nullptr, w);
  }
  cudaStreamSynchronize(s);
  cudaFree(w);
  cudaFree(m);
  CK(e);
  OP_END();
}

int ib_op_cn_a(ib_handle* h, int32_t lev, const double* b, double* x) { return cn_op(h, lev, b, x, false); }
int ib_op_cn_ainv(ib_handle* h, int32_t lev, const double* b, double* x) { return cn_op(h, lev, b, x, true); }

int ib_op_curl(ib_handle* h, const double* psi, const double* bc, double* q) {
  OP_BEGIN();
  CK(curl<double>(g, psi, bc, q, 1, s));
  OP_END();
}

int ib_op_rot(ib_handle* h, const double* q, double* gamma) {
  OP_BEGIN();
  CK(rot<double>(g, q, gamma, 1, s));
  OP_END();
}

int ib_op_coarsify(ib_handle* h, double* gc, const double* gf) {
  OP_BEGIN();
  CK(coarsify<double>(g, gc, gf, 1, g.nG, s));
  OP_END();
}

int ib_op_get_bc(ib_handle* h, const double* r, double* bc) {
  OP_BEGIN();
  CK(get_bc<double>(g, r, bc, 1, 1.0, s));
  OP_END();
}

int ib_op_apply_bc(ib_handle* h, double* r, const double* bc, double fac) {
  OP_BEGIN();
  CK(apply_bc<double>(g, r, bc, fac, 1, s));
  OP_END();
}

int ib_op_nonlinear(ib_handle* h, int32_t lev, const double* q, double u, double v, const double* gamma,
                    const double* bc, double* nonlin) {
  OP_BEGIN();
  if (lev < 1 || lev > g.nlev) return IB_ERR_INVALID;
  Geometry g1 = g;
  g1.nlev = 1;
  const double hc = g.h * std::ldexp(1.0, lev - 1);
  double par[3] = {u * hc, v * hc, 1.0 / (hc * hc)};
  double *dpar, *zero_ring, *zero_g, *scratch, *edges;
  const int ne = 2 * (g.nx - 1) + 2 * (g.ny - 1);
  CK(cudaMalloc(&dpar, sizeof(par)));
  CK(cudaMalloc(&zero_ring, sizeof(double) * g.nbc));
  CK(cudaMalloc(&zero_g, sizeof(double) * g.nG));
  CK(cudaMalloc(&scratch, sizeof(double) * g.nG));
  CK(cudaMalloc(&edges, sizeof(double) * ne));
  CK(cudaMemcpyAsync(dpar, par, sizeof(par), cudaMemcpyHostToDevice, s));
  CK(cudaMemsetAsync(zero_ring, 0, sizeof(double) * g.nbc, s));
  CK(cudaMemsetAsync(zero_g, 0, sizeof(double) * g.nG, s));
  CK(cudaMemsetAsync(edges, 0, sizeof(double) * ne, s));
  NonlinArgs<double> na{};
  na.q = q;
  na.gamma = gamma;
  na.bcn = bc ? bc : zero_ring;
  na.nl_old = zero_g;
  na.edges = edges;
  na.nl_new = nonlin;
  na.rhs = scratch;
  na.q0 = dpar;
  na.inv_hc2 = dpar + 2;
  na.dtb0 = 0.0;
  na.dtb1 = 0.0;
  cudaError_t e = nonlin_rhs<double>(g1, na, s);
  cudaStreamSynchronize(s);
  cudaFree(dpar); cudaFree(zero_ring); cudaFree(zero_g); cudaFree(scratch); cudaFree(edges);
  CK(e);
  OP_END();
}

int ib_op_vort2flux(ib_handle* h, double* gamma, double* psi, double* q) {
  OP_BEGIN();
  OpWork work(h);
  double* rings;
  CK(work.get(&rings, (int64_t)g.nlev * g.nbc));
  cudaError_t e = vort2flux<double>(h, gamma, psi, q, nullptr, rings);
  work.done();
  CK(e);
  OP_END();
}

int ib_op_reg_gather(ib_handle* h, const double* q, double u, double v, double* fb) {
  OP_BEGIN();
  if (h->nb == 0) return IB_OK;
  double par[2] = {u * g.h, v * g.h};
  double* dpar;
  CK(cudaMalloc(&dpar, sizeof(par)));
  CK(cudaMemcpyAsync(dpar, par, sizeof(par), cudaMemcpyHostToDevice, s));
  cudaError_t e = reg_gather<double>(g, q, dpar, h->body_idx, h->weight, h->nb, fb, 1, g.nq, h->nf, s);
  cudaStreamSynchronize(s);
  cudaFree(dpar);
  CK(e);
  OP_END();
}

int ib_op_reg_scatter(ib_handle* h, const double* fb, double* q) {
  OP_BEGIN();
  CK(cudaMemsetAsync(q, 0, sizeof(double) * g.nq, s));
  if (h->nb == 0) { OP_END(); }
  CK(reg_scatter<double>(g, fb, h->body_idx, h->weight, h->nb, q, h->status + 1, s));
  CK(cudaStreamSynchronize(s));
  return check_status(h);
}

int ib_get_schur(ib_handle* h, double* bmat, double* binv) {
  OP_BEGIN();
  const size_t bytes = sizeof(double) * (size_t)h->nf * h->nf;
  if (h->nf == 0) return IB_OK;
  if (!h->bmat) return fail(h, IB_ERR_INVALID, "no assembled Schur matrix (moving bodies without preconditioner)");
  if (bmat) CK(cudaMemcpyAsync(bmat, h->bmat, bytes, cudaMemcpyDeviceToHost, s));
  if (binv) CK(cudaMemcpyAsync(binv, h->binv_cm, bytes, cudaMemcpyDeviceToHost, s));
  OP_END();
}

int ib_get_reg(ib_handle* h, int32_t* body_idx, double* weight) {
  OP_BEGIN();
  if (h->nb == 0) return IB_OK;
  if (body_idx) CK(cudaMemcpyAsync(body_idx, h->body_idx, sizeof(int) * 2 * h->nb, cudaMemcpyDeviceToHost, s));
  if (weight) CK(cudaMemcpyAsync(weight, h->weight, sizeof(double) * h->nb * 2 * kWin2, cudaMemcpyDeviceToHost, s));
  OP_END();
}

// ------------------------------------------------------------------------------------------------
// learned warm start (include/ibgb300_learn.h)
// ------------------------------------------------------------------------------------------------
int ib_learn_init(ib_handle* h, int32_t hidden, int32_t hidden_layers, int32_t capacity, uint64_t seed) {
  if (!h) return IB_ERR_INVALID;
  if (h->motion != IB_MOTION_PRESCRIBED || h->nf == 0)
    return fail(h, IB_ERR_INVALID, "the learned warm start needs moving bodies");
  if (hidden < 1 || hidden > 4096 || hidden_layers < 1 || hidden_layers > 8 || capacity < 2 || capacity > (1 << 20))
    return fail(h, IB_ERR_INVALID, "network size or sample capacity out of range");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  delete h->mlp;
  h->mlp = new learn::Mlp();
  const int din = 6 * h->nbodies + 2 * h->nf;
  cudaError_t e = h->mlp->init(din, h->nf, hidden, hidden_layers, capacity, seed, h->stream, h->status + 3);
  if (e != cudaSuccess) {
    delete h->mlp;
    h->mlp = nullptr;
    return fail(h, IB_ERR_CUDA, "network allocation", e);
  }
  return IB_OK;
}

int ib_learn_collect(ib_handle* h, int32_t on) {
  if (!h || !h->mlp) return h ? fail(h, IB_ERR_INVALID, "no network (ib_learn_init)") : IB_ERR_INVALID;
  h->collect = on != 0;
  return IB_OK;
}

int ib_learn_sample_count(ib_handle* h, int32_t* count) {
  if (!h || !count) return IB_ERR_INVALID;
  *count = h->mlp ? h->mlp->count : 0;
  return IB_OK;
}

int ib_learn_train(ib_handle* h, int32_t epochs, int32_t batch, double lr, uint64_t seed, double* final_loss) {
  ib::Range nvtx_range("ib_learn_train");
  if (!h || !h->mlp) return h ? fail(h, IB_ERR_INVALID, "no network (ib_learn_init)") : IB_ERR_INVALID;
  if (epochs < 1 || batch < 1 || batch > learn::kMaxBatch || !(lr > 0))
    return fail(h, IB_ERR_INVALID, "epochs, batch (1..512) and learning rate must be positive");
  if (h->mlp->count < 2) return fail(h, IB_ERR_INVALID, "fewer than two recorded samples");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  cudaError_t e = h->mlp->train(epochs, batch, (float)lr, seed, final_loss);
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "training", e);
  if (h->mlp->val_rows.empty()) return IB_OK;
  return h->precision == IB_PREC_MIXED ? learn_validate_schur<df64>(h) : learn_validate_schur<double>(h);
}

int ib_learn_validation(ib_handle* h, double* blend, double* rel_err) {
  if (!h || !h->mlp) return IB_ERR_INVALID;
  if (blend) *blend = h->mlp->blend;
  if (rel_err) *rel_err = h->mlp->val_rel;
  return IB_OK;
}

int ib_learn_layout(ib_handle* h, int32_t* nlayers, int32_t* dims, int32_t max_dims) {
  if (!h || !h->mlp || !nlayers) return IB_ERR_INVALID;
  *nlayers = h->mlp->nl;
  if (dims)
    for (int i = 0; i <= h->mlp->nl && i < max_dims; ++i) dims[i] = h->mlp->dims[i];
  return IB_OK;
}

int ib_learn_param_count(ib_handle* h, int64_t* nparam) {
  if (!h || !h->mlp || !nparam) return IB_ERR_INVALID;
  *nparam = h->mlp->nparam;
  return IB_OK;
}

int ib_learn_get_params(ib_handle* h, float* params) {
  if (!h || !h->mlp || !params) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  CK(cudaMemcpyAsync(params, h->mlp->master, sizeof(float) * h->mlp->nparam, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return IB_OK;
}

int ib_learn_set_params(ib_handle* h, const float* params) {
  if (!h || !h->mlp || !params) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  CK(cudaMemcpyAsync(h->mlp->master, params, sizeof(float) * h->mlp->nparam, cudaMemcpyHostToDevice, h->stream));
  CK(h->mlp->sync_bf16());
  CK(cudaStreamSynchronize(h->stream));
  return IB_OK;
}

int ib_learn_set_blend(ib_handle* h, double blend) {
  if (!h || !h->mlp || !(blend >= 0.0 && blend <= 1.0)) return IB_ERR_INVALID;
  h->mlp->blend = blend;
  // the captured moving step holds the blend as a kernel argument: capture it again
  for (auto& ge : h->mgexec)
    if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
  return IB_OK;
}

int ib_learn_export(ib_handle* h, float* buf, int64_t n) {
  if (!h || !h->mlp || !buf) return IB_ERR_INVALID;
  learn::Mlp* m = h->mlp;
  const int din = m->dims[0], dout = m->dims[m->nl];
  if (n != m->nparam + 2 * (int64_t)din + 2 * (int64_t)dout + 1) return fail(h, IB_ERR_INVALID, "learn export: size");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  cudaStream_t s = h->stream;
  float* p = buf;
  CK(cudaMemcpyAsync(p, m->master, sizeof(float) * m->nparam, cudaMemcpyDeviceToHost, s)); p += m->nparam;
  CK(cudaMemcpyAsync(p, m->mu_x, sizeof(float) * din, cudaMemcpyDeviceToHost, s)); p += din;
  CK(cudaMemcpyAsync(p, m->sd_x, sizeof(float) * din, cudaMemcpyDeviceToHost, s)); p += din;
  CK(cudaMemcpyAsync(p, m->mu_y, sizeof(float) * dout, cudaMemcpyDeviceToHost, s)); p += dout;
  CK(cudaMemcpyAsync(p, m->sd_y, sizeof(float) * dout, cudaMemcpyDeviceToHost, s)); p += dout;
  CK(cudaStreamSynchronize(s));
  *p = (float)m->blend;
  return IB_OK;
}

int ib_learn_import(ib_handle* h, const float* buf, int64_t n) {
  if (!h || !h->mlp || !buf) return IB_ERR_INVALID;
  learn::Mlp* m = h->mlp;
  const int din = m->dims[0], dout = m->dims[m->nl];
  if (n != m->nparam + 2 * (int64_t)din + 2 * (int64_t)dout + 1) return fail(h, IB_ERR_INVALID, "learn import: size");
  const double blend = buf[n - 1];
  if (!(blend >= 0.0 && blend <= 1.0)) return fail(h, IB_ERR_INVALID, "learn import: blend outside [0, 1]");
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  cudaStream_t s = h->stream;
  const float* p = buf;
  CK(cudaMemcpyAsync(m->master, p, sizeof(float) * m->nparam, cudaMemcpyHostToDevice, s)); p += m->nparam;
  CK(cudaMemcpyAsync(m->mu_x, p, sizeof(float) * din, cudaMemcpyHostToDevice, s)); p += din;
  CK(cudaMemcpyAsync(m->sd_x, p, sizeof(float) * din, cudaMemcpyHostToDevice, s)); p += din;
  CK(cudaMemcpyAsync(m->mu_y, p, sizeof(float) * dout, cudaMemcpyHostToDevice, s)); p += dout;
  CK(cudaMemcpyAsync(m->sd_y, p, sizeof(float) * dout, cudaMemcpyHostToDevice, s)); p += dout;
  CK(m->sync_bf16());
  CK(cudaStreamSynchronize(s));
  m->blend = blend;
  m->trained = true;
  for (auto& ge : h->mgexec)
    if (ge) { cudaGraphExecDestroy(ge); ge = nullptr; }
  return IB_OK;
}

int ib_learn_gradients(ib_handle* h, int32_t rows, const float* x, const float* y, float* grad, double* loss) {
  if (!h || !h->mlp || !x || !y || rows < 1 || rows > learn::kMaxBatch) return IB_ERR_INVALID;
  DeviceGuard dev_guard_(h->device);
  CK(dev_guard_.err);
  cudaError_t e = h->mlp->gradients(rows, x, y, grad, loss);
  if (e != cudaSuccess) return fail(h, IB_ERR_CUDA, "network gradients", e);
  return IB_OK;
}

int ib_get_cg_start_residuals(ib_handle* h, int32_t count, double* r0) {
  if (!h || count < 0 || count > (int32_t)h->cg_res0.size()) return IB_ERR_INVALID;
  const size_t off = h->cg_res0.size() - (size_t)count;
  for (int i = 0; i < count; ++i)
    if (r0) r0[i] = h->cg_res0[off + i];
  return IB_OK;
}

// ------------------------------------------------------------------------------------------------
// ensembles (include/ibgb300_ensemble.h)
// ------------------------------------------------------------------------------------------------
}  // extern "C"

struct ib_ensemble {
  int device = 0;
  std::vector<ib_handle*> m;
  cudaStream_t stream = nullptr;
  cudaEvent_t start = nullptr;
  std::vector<cudaEvent_t> join;
  cudaGraphExec_t gexec[2] = {nullptr, nullptr};    // one step, per starting parity
  cudaGraphExec_t gexec_k[2] = {nullptr, nullptr};  // `chunk` steps, per starting parity
  int chunk = 1;                                    // steps per launch (ib_ensemble_set_steps_per_launch)
  double* h_q0 = nullptr;  // pinned [2][kMaxStepsPerLaunch][slot_len]: base flux of every member and level
  std::vector<int64_t> q0_off;
  int64_t slot_len = 0;
  cudaEvent_t done[2] = {nullptr, nullptr};
  bool launched[2] = {false, false};
  int parity = 0;
  int kernels_per_step = 0;
  bool any_moving = false;
  std::vector<uint64_t> keys;        // moving members' capture keys at capture time
  std::string err;
};

namespace {

int efail(ib_ensemble* e, int code, const std::string& what, cudaError_t ce = cudaSuccess) {
  std::string msg = what;
  if (ce != cudaSuccess) {
    msg += ": ";
    msg += cudaGetErrorString(ce);
  }
  if (e) e->err = msg;
  else {
    std::lock_guard<std::mutex> lock(g_err_mu);
    g_create_err = msg;
  }
  return code;
}

#define EK(x)                                                              \
  do {                                                                     \
    cudaError_t e_ = (x);                                                  \
    if (e_ != cudaSuccess) return efail(e, IB_ERR_CUDA, #x, e_);           \
  } while (0)

void destroy_ensemble(ib_ensemble* e) {
  if (!e) return;
  DeviceGuard dev_guard_(e->device);
  if (e->stream) cudaStreamSynchronize(e->stream);
  for (auto& g : e->gexec)
    if (g) cudaGraphExecDestroy(g);
  for (auto& g : e->gexec_k)
    if (g) cudaGraphExecDestroy(g);
  for (auto ev : e->join)
    if (ev) cudaEventDestroy(ev);
  for (auto ev : e->done)
    if (ev) cudaEventDestroy(ev);
  if (e->start) cudaEventDestroy(e->start);
  if (e->h_q0) cudaFreeHost(e->h_q0);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
}

// capture `nsteps` ensemble steps for launches at ensemble parity p, reading staging slot set p;
// member i runs its parities base_i ^ p, base_i ^ p ^ 1, ..., base_i being its parity at ensemble
// parity 0 (its current parity is base_i ^ e->parity).  Each member's steps follow one another
// on its own branch and the branches join only at the end, so within one launch a member does
// not wait for the others.
int capture_ensemble(ib_ensemble* e, int p, int nsteps = 1) {
  cudaGraph_t graph = nullptr;
  EK(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
  cudaError_t ce = cudaEventRecord(e->start, e->stream);
  for (size_t i = 0; i < e->m.size() && ce == cudaSuccess; ++i) {
    ib_handle* h = e->m[i];
    ce = cudaStreamWaitEvent(h->stream, e->start, 0);
    for (int k = 0; k < nsteps && ce == cudaSuccess; ++k) {
      const int par = h->parity ^ e->parity ^ p ^ (k & 1);
      if (h->motion == IB_MOTION_PRESCRIBED) {
        // the member's own staging slot k holds this step's base flux and kinematics
        ce = h->precision == IB_PREC_MIXED ? enqueue_moving_captured<df64>(h, par, k)
                                           : enqueue_moving_captured<double>(h, par, k);
      } else {
        const double* slot = e->h_q0 + ((size_t)p * kMaxStepsPerLaunch + k) * e->slot_len + e->q0_off[i];
        ce = cudaMemcpyAsync(h->d_q0, slot, sizeof(double) * 2 * h->g.nlev, cudaMemcpyHostToDevice, h->stream);
        if (ce == cudaSuccess) ce = enqueue_step_mode(h, par);
      }
    }
    if (ce == cudaSuccess) ce = cudaEventRecord(e->join[i], h->stream);
    if (ce == cudaSuccess) ce = cudaStreamWaitEvent(e->stream, e->join[i], 0);
  }
  cudaError_t ce2 = cudaStreamEndCapture(e->stream, &graph);
  if (ce != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    return efail(e, IB_ERR_CUDA, "ensemble capture", ce);
  }
  if (ce2 != cudaSuccess) return efail(e, IB_ERR_CUDA, "ensemble capture", ce2);
  size_t nn = 0;
  if (cudaGraphGetNodes(graph, nullptr, &nn) == cudaSuccess && nn > 0) {
    std::vector<cudaGraphNode_t> nodes(nn);
    cudaGraphGetNodes(graph, nodes.data(), &nn);
    int k = 0;
    for (auto nd : nodes) {
      cudaGraphNodeType ty;
      if (cudaGraphNodeGetType(nd, &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel) ++k;
    }
    if (nsteps == 1) e->kernels_per_step = k;
  }
  cudaGraphExec_t& slot_exec = nsteps == 1 ? e->gexec[p] : e->gexec_k[p];
  if (slot_exec) {
    cudaGraphExecDestroy(slot_exec);
    slot_exec = nullptr;
  }
  ce = cudaGraphInstantiate(&slot_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess) return efail(e, IB_ERR_CUDA, "ensemble graph instantiate", ce);
  return IB_OK;
}

}  // namespace

extern "C" {

int ib_ensemble_create(ib_handle* const* members, int32_t n, ib_ensemble** out) {
  if (!members || n < 1 || !out) return efail(nullptr, IB_ERR_INVALID, "ensemble: no members");
  *out = nullptr;
  for (int i = 0; i < n; ++i) {
    const ib_handle* h = members[i];
    if (!h) return efail(nullptr, IB_ERR_INVALID, "ensemble: null member");
    if (h->motion == IB_MOTION_PRESCRIBED &&
        (!h->use_moving_graph || h->steps < 2 || (h->precond == IB_PC_SCHUR_REF && h->pc_step < 0)))
      return efail(nullptr, IB_ERR_UNSUPPORTED,
                   "a moving member joins after its first two steps (and first preconditioner), with graphs enabled");
    if (h->device != members[0]->device || h->steps != members[0]->steps)
      return efail(nullptr, IB_ERR_INVALID, "ensemble members must share the device and the step count");
    for (int j = 0; j < i; ++j)
      if (members[j] == h) return efail(nullptr, IB_ERR_INVALID, "ensemble member given twice");
  }
  DeviceGuard dev_guard_(members[0]->device);
  ib_ensemble* e = new ib_ensemble();
  e->device = members[0]->device;
  e->m.assign(members, members + n);
  cudaError_t ce = dev_guard_.err;
  auto bail = [&](int rc) {
    {
      std::lock_guard<std::mutex> lock(g_err_mu);
      g_create_err = e->err;
    }
    destroy_ensemble(e);
    return rc;
  };
  if (ce != cudaSuccess) return bail(efail(e, IB_ERR_CUDA, "cudaSetDevice", ce));
  // static members fill the GPU between them: the level-by-level Vort2Flux there
  if (n >= 2)
    for (ib_handle* h : e->m)
      if (h->motion != IB_MOTION_PRESCRIBED && h->precision == IB_PREC_MIXED && h->v2f_levels && !h->v2f_fx) {
        const int rc = ib_set_vort2flux_order(h, IB_V2F_SEQUENTIAL);
        if (rc != IB_OK) return bail(efail(e, rc, "member Vort2Flux order: " + h->err));
      }
  for (ib_handle* h : e->m) {
    if (h->motion == IB_MOTION_PRESCRIBED) {
      e->any_moving = true;
      e->keys.push_back(moving_graph_key(h));
    } else {
      e->keys.push_back(0);
    }
    e->q0_off.push_back(e->slot_len);
    e->slot_len += 2 * h->g.nlev;
    if ((ce = cudaStreamSynchronize(h->stream)) != cudaSuccess) return bail(efail(e, IB_ERR_CUDA, "member sync", ce));
  }
  if ((ce = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking)) != cudaSuccess) {
    e->stream = nullptr;
    return bail(efail(e, IB_ERR_CUDA, "cudaStreamCreate", ce));
  }
  if ((ce = cudaEventCreateWithFlags(&e->start, cudaEventDisableTiming)) != cudaSuccess) {
    e->start = nullptr;
    return bail(efail(e, IB_ERR_CUDA, "cudaEventCreate", ce));
  }
  e->join.assign(n, nullptr);
  for (auto& ev : e->join)
    if ((ce = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
      ev = nullptr;
      return bail(efail(e, IB_ERR_CUDA, "cudaEventCreate", ce));
    }
  for (auto& ev : e->done)
    if ((ce = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
      ev = nullptr;
      return bail(efail(e, IB_ERR_CUDA, "cudaEventCreate", ce));
    }
  if ((ce = cudaMallocHost(&e->h_q0, sizeof(double) * 2 * kMaxStepsPerLaunch * (size_t)e->slot_len)) != cudaSuccess) {
    e->h_q0 = nullptr;
    return bail(efail(e, IB_ERR_CUDA, "pinned staging", ce));
  }
  for (int p = 0; p < 2; ++p) {
    int rc = capture_ensemble(e, p);
    if (rc != IB_OK) return bail(rc);
  }
  *out = e;
  return IB_OK;
}

int ib_ensemble_destroy(ib_ensemble* e) {
  destroy_ensemble(e);
  return IB_OK;
}

int ib_ensemble_advance_n(ib_ensemble* e, int32_t nsteps, const double* t, const double* uv, double* device_ms) {
  ib::Range nvtx_range("ib_ensemble_advance_n");
  if (e && e->any_moving) return efail(e, IB_ERR_INVALID, "moving members need kinematics (ib_ensemble_advance_n_kin)");
  return ib_ensemble_advance_n_kin(e, nsteps, t, uv, nullptr, device_ms);
}

int ib_ensemble_advance_n_kin(ib_ensemble* e, int32_t nsteps, const double* t, const double* uv, const double* kin,
                              double* device_ms) {
  ib::Range nvtx_range("ib_ensemble_advance_n_kin");
  if (!e || nsteps < 0 || (nsteps > 0 && (!t || !uv))) return IB_ERR_INVALID;
  if (e->any_moving && nsteps > 0 && !kin) return efail(e, IB_ERR_INVALID, "moving members need kinematics");
  DeviceGuard dev_guard_(e->device);
  EK(dev_guard_.err);
  int kin_per_step = 0;
  for (ib_handle* h : e->m)
    if (h->motion == IB_MOTION_PRESCRIBED) kin_per_step += 6 * h->nbodies;
  const int n = (int)e->m.size();
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (device_ms) {
    EK(cudaEventCreate(&e0));
    EK(cudaEventCreate(&e1));
    EK(cudaEventRecord(e0, e->stream));
  }
  for (int s = 0; s < nsteps;) {
    const int K = (e->chunk > 1 && nsteps - s >= e->chunk) ? e->chunk : 1;
    const int p = e->parity;
    // the launch that read slot set p last must be done before the set is rewritten
    if (e->launched[p]) EK(cudaEventSynchronize(e->done[p]));
    for (int k = 0; k < K; ++k) {
      double* slot = e->h_q0 + ((size_t)p * kMaxStepsPerLaunch + k) * e->slot_len;
      const double* ks = kin ? kin + (size_t)(s + k) * kin_per_step : nullptr;
      for (int i = 0; i < n; ++i) {
        ib_handle* h = e->m[i];
        const double u = uv[((size_t)(s + k) * n + i) * 2], v = uv[((size_t)(s + k) * n + i) * 2 + 1];
        const bool mv = h->motion == IB_MOTION_PRESCRIBED;
        double* dst = mv ? h->h_mslot + (size_t)k * (2 * h->g.nlev + 6 * h->nbodies) : slot + e->q0_off[i];
        for (int l = 0; l < h->g.nlev; ++l) {
          const double hc = h->g.h * std::ldexp(1.0, l);  // base_flux!, fluid-ops.jl:414-415
          dst[2 * l] = u * hc;
          dst[2 * l + 1] = v * hc;
        }
        if (mv) {
          std::memcpy(dst + 2 * h->g.nlev, ks, sizeof(double) * 6 * h->nbodies);
          ks += 6 * h->nbodies;
        }
      }
    }
    for (int i = 0; i < n; ++i) {
      ib_handle* h = e->m[i];
      if (h->motion != IB_MOTION_PRESCRIBED) continue;
      // preconditioner re-assembly between launches, on the member's own stream
      int rc = pc_maybe_assemble(h);
      if (rc != IB_OK) return efail(e, rc, "member " + std::to_string(i) + ": " + h->err);
      if (moving_graph_key(h) != e->keys[i])
        return efail(e, IB_ERR_INVALID, "member " + std::to_string(i) + " changed its CG options inside the ensemble");
    }
    EK(cudaGraphLaunch(K == 1 ? e->gexec[p] : e->gexec_k[p], e->stream));
    EK(cudaEventRecord(e->done[p], e->stream));
    e->launched[p] = true;
    e->parity ^= K & 1;
    if (e->any_moving) {
      // moving members: the steps' CG statistics came back through pinned memory
      EK(cudaStreamSynchronize(e->stream));
      for (int i = 0; i < n; ++i) {
        ib_handle* h = e->m[i];
        if (h->motion != IB_MOTION_PRESCRIBED) continue;
        for (int k = 0; k < K; ++k) {
          const double* o = h->h_cgout + 4 * k;
          h->cg_iters.push_back((int)o[0]);
          h->cg_res.push_back(o[1]);
          h->cg_res0.push_back(o[2]);
          if (h->mlp && h->collect) h->mlp->record_commit();
          pc_account(h, h->steps + k);
          if (o[3] != 0.0)
            return efail(e, IB_ERR_CG_MAXITER, "member " + std::to_string(i) + ": Schur CG iteration cap");
        }
      }
    }
    for (int i = 0; i < n; ++i) {
      ib_handle* h = e->m[i];
      h->parity ^= K & 1;
      h->steps += K;
      h->t = t[(size_t)(s + K - 1) * n + i];
    }
    s += K;
  }
  if (device_ms) {
    EK(cudaEventRecord(e1, e->stream));
    EK(cudaEventSynchronize(e1));
    float ms = 0.f;
    EK(cudaEventElapsedTime(&ms, e0, e1));
    *device_ms = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  EK(cudaStreamSynchronize(e->stream));
  for (int i = 0; i < n; ++i) {
    int rc = check_status(e->m[i]);
    if (rc != IB_OK) return efail(e, rc, "member " + std::to_string(i) + ": " + e->m[i]->err);
  }
  return IB_OK;
}

int ib_ensemble_set_steps_per_launch(ib_ensemble* e, int32_t k) {
  ib::Range nvtx_range("ib_ensemble_set_steps_per_launch");
  if (!e) return IB_ERR_INVALID;
  if (k < 1 || k > kMaxStepsPerLaunch)
    return efail(e, IB_ERR_INVALID, "steps per launch must be 1.." + std::to_string(kMaxStepsPerLaunch));
  DeviceGuard dev_guard_(e->device);
  EK(dev_guard_.err);
  EK(cudaStreamSynchronize(e->stream));
  for (auto& g : e->gexec_k)
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
  e->chunk = k;
  if (k == 1) return IB_OK;
  for (int p = 0; p < 2; ++p) {
    const int rc = capture_ensemble(e, p, k);
    if (rc != IB_OK) {
      e->chunk = 1;
      return rc;
    }
  }
  return IB_OK;
}

int ib_ensemble_info(ib_ensemble* e, int32_t* members, int32_t* kernels_per_step) {
  if (!e) return IB_ERR_INVALID;
  if (members) *members = (int32_t)e->m.size();
  if (kernels_per_step) *kernels_per_step = e->kernels_per_step;
  return IB_OK;
}

const char* ib_ensemble_last_error(const ib_ensemble* e) {
  if (e) return e->err.c_str();
  std::lock_guard<std::mutex> lock(g_err_mu);
  return g_create_err.c_str();
}

}  // extern "C"
