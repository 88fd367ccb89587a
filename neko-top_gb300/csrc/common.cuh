// Shared definitions of the GB300 SEM library: error handling, the plan
// structure, device scalar block and deterministic reductions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ntgb300.h"

#define NTG_LXMAX 12

namespace ntg {

void set_error(const char* fmt, ...);
void clear_error();

// Returns NTG_ERR_CUDA (and records the message) if a CUDA call failed.
#define NTG_CUDA_TRY(call)                                                             \
  do {                                                                                 \
    cudaError_t _e = (call);                                                           \
    if (_e != cudaSuccess) {                                                           \
      ::ntg::set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(_e)); \
      return NTG_ERR_CUDA;                                                             \
    }                                                                                  \
  } while (0)

#define NTG_CHECK_ARG(cond, msg)            \
  do {                                      \
    if (!(cond)) {                          \
      ::ntg::set_error("%s", msg);          \
      return NTG_ERR_INVALID;               \
    }                                       \
  } while (0)

#define NTG_TRY(expr)              \
  do {                             \
    int _s = (expr);               \
    if (_s != NTG_OK) return _s;   \
  } while (0)

template <typename T>
int dev_alloc(T** p, size_t count) {
  *p = nullptr;
  if (count == 0) return NTG_OK;
  cudaError_t e = cudaMalloc((void**)p, sizeof(T) * count);
  if (e != cudaSuccess) {
    set_error("cudaMalloc of %zu bytes failed: %s", sizeof(T) * count, cudaGetErrorString(e));
    *p = nullptr;
    return NTG_ERR_ALLOC;
  }
  return NTG_OK;
}
template <typename T>
void dev_free(T*& p) {
  if (p) cudaFree(p);
  p = nullptr;
}

// Partial-sum slots of the deterministic two-level reductions: each block
// writes its partial to part[blockIdx.x]; the last block to finish (found
// with an atomic ticket) sums part[0..gridDim.x) in index order.
constexpr int kRedSlots = 4096;   // max blocks of a reducing kernel
constexpr int kRedLanes = 32;     // up to 32 simultaneous sums per kernel

// Device-resident solver scalars (one block per solve, FP64).
struct Scalars {
  double rz;       // (r, z) of the current iteration
  double rz_new;
  double pap;      // (p, Ap)
  double alpha, beta;
  double rr;       // (r, r) mult-weighted
  double tol2;     // squared stopping threshold
  double ff;       // (f, f)
  double rtol, abstol;
  double pap_prev; // (p_{k-1}, A p_{k-1}) of the flexible CG
  double gamma;    // flexible-CG orthogonalisation coefficient
  double rr0;      // (r0, r0) at the start of the solve
  double rmax;     // reliable updates: largest ||r|| since the last FP64 residual
  double delta;    // reliable updates: replace the residual when ||r|| < delta * rmax
  double red[8];   // scratch results of generic reductions
  int ru_mode;     // 1 = FP32 iteration with FP64 reliable updates
  int need_ru;     // 1 = residual replacement due, 2 = FP32 residual converged (confirm in FP64)
  int ext_pc;      // 1 = preconditioner applied by separate kernels: (r, z) and beta come from k_rz
  int y_due;       // the last update's y += alpha p is still to be done (AxDir or k_ru_accum)
  int iter;        // iterations performed
  int done;        // 1 = converged or stopped: later kernels are no-ops
  int status;      // NTG_OK / NTG_MAXITER / NTG_BREAKDOWN / NTG_NONFINITE
  int max_iter;
  unsigned ticket; // last-block ticket of the reducing kernels
  unsigned pad;
};

}  // namespace ntg

// The Dirichlet mask and what is derived from it.  One object, so that a mask
// that is set aside for a while (ntg_filter_apply) takes all of it along.
struct ntg_mask_state {
  int32_t* mask = nullptr;      // 0-based node list
  int64_t nmask = 0;
  uint8_t* maskrow = nullptr;   // n / lx (lx <= 8): bit i of byte t set when node i of row t is masked; null: no mask
  double* multm = nullptr;      // mult, negative on Dirichlet nodes (plan_multm; null until used)
  float* multmf = nullptr;      // multf, likewise
};

// The plan: mesh, coef_t, gs_t, Jacobi, the Dirichlet mask.
struct ntg_plan : ntg_mask_state {
  int lx = 0;
  int64_t nelv = 0, n = 0, nu = 0, nshared = 0, nshared_idx = 0;
  cudaStream_t stream = 0;
  double D[NTG_LXMAX * NTG_LXMAX];
  double wq[NTG_LXMAX];
  float Df[NTG_LXMAX * NTG_LXMAX];
  // geometry (FP64 + FP32 copies)
  double* g[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  float* gf[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  double* B = nullptr;
  double* mult = nullptr;
  float* multf = nullptr;
  // gather-scatter: full map (perm sorted by global id, offsets) and the
  // shared-node subset the hot kernels use
  int32_t* perm = nullptr;
  int64_t* offs = nullptr;
  int32_t* sh_idx = nullptr;  // local indices of nodes with > 1 copy, grouped
  int32_t* sh_off = nullptr;  // nshared + 1 offsets into sh_idx
  // the same groups split by multiplicity (2, 4, 8, other), each class
  // ordered by its first local index (gs_classes.cu)
  int gs_classes = 1;           // 1: class kernel (default); 0: one thread per group
  int64_t ncls[4] = {0, 0, 0, 0};
  int2* gs2 = nullptr;
  int4* gs4 = nullptr;
  int4* gs8 = nullptr;          // two int4 per group
  int32_t* gsx_idx = nullptr;
  int32_t* gsx_off = nullptr;
  // coefficients
  int h1_const = 1;
  double h1c = 1.0;
  double* h1 = nullptr;   // n (when !h1_const)
  float* h1f = nullptr;
  int ifh2 = 0;
  double* hB = nullptr;   // h2*B (when ifh2)
  float* hBf = nullptr;
  // Jacobi
  double* dinv = nullptr;
  float* dinvf = nullptr;
  int jacobi_ready = 0;
  // FP32 Ax path: 1 = bulk-copy pipelined kernel for lx = 8 (default)
  int use_tma = 1;
  int* dev_err = nullptr;        // set by kernels whose bounded waits ran out
  // reductions
  double* red_part = nullptr;    // kRedSlots * kRedLanes
  ntg::Scalars* scal = nullptr;  // generic scalars for standalone dots
  double* host_red = nullptr;    // pinned
  // derivative operators (deriv.cu): 9 metric cofactors and 1/jac
  // (10 x n), and 1 / gs(B)
  double* met = nullptr;
  double* binv = nullptr;
  double* dscr = nullptr;  // their scratch (plan_scratch)
  int64_t dscr_n = 0;
  // fixed-point forms of D and D^T (fx.cuh), made on first use
  struct FxCache {
    std::mutex mu;
    struct Entry {
      double scale;
      bool weighted;
      std::shared_ptr<void> mats;
    };
    std::vector<Entry> mats;
  };
  std::unique_ptr<FxCache> fx{new FxCache};
};

namespace ntg {
// Every kernel launch of the library bumps this counter (read through
// ntg_launch_count); it is how callers count the library's launches.
void count_launch();
#define NTG_COUNT_LAUNCH() ::ntg::count_launch()

// Optional per-kernel device timers (CUDA events on the launching stream),
// off by default; enabled with ntg_timer_enable.
enum TimerId {
  TM_AX64 = 0, TM_AX32 = 1, TM_GS64 = 2, TM_GS32 = 3, TM_UPD64 = 4, TM_UPD32 = 5, TM_DIR64 = 6,
  TM_DIR32 = 7, TM_PC32 = 8, TM_FDM = 9, TM_CRS = 10, TM_PULL = 11, TM_COUNT = 16
};
// z = M r with the Schwarz preconditioner (schwarz.cu); no-op once sc->done
// z = M r (FP32).  With mult non-null also (r, z)_mult into sc (FinRz{rz_mode}).
int schwarz_apply(ntg_schwarz* sw, float* z, const float* r, cudaStream_t s, Scalars* sc, const float* mult = nullptr,
                  double* part = nullptr, int rz_mode = 0);
void timer_start(int id, cudaStream_t s);
void timer_stop(int id, cudaStream_t s);

// Programmatic dependent launch for the kernels of the solver iterations: on
// small meshes they take 3 to 20 us each, one after another, and most of that
// is the launch and the last blocks of the kernel before.  A kernel that begins
// with dependent_wait() may be launched by launch_dependent() while its
// predecessor still runs: it waits for the predecessor's end (which waited for
// everything before it) before it touches memory.  (Exceptions, each with its
// reason: the coarse solve's matrices and stop flag.)  dependent_start() also
// lets the successor be scheduled.  k_fdm leaves that out (0.4% of a solve at 43M
// nodes for the instruction alone; the coarse solve relies on it), and the FP64
// operator takes no part: with its successors waiting beside it an FP64 solve at
// 0.26M nodes went from 38.7 to 43.9 ms, without from 38.7 to 35.1.
//
// The waiting blocks take room from the kernel that runs, so from some size on
// they cost more than the launches they hide.  Measured with and without, one
// FP32 operator and preconditioner at lx = 8: 28.6 and 45.1 us at 0.26M nodes,
// 58 and 70 us at 1M; a mixed Poisson solve: 7.6 and 9.5 ms at 2.1M, 12.0 and
// 14.0 ms at 4.2M; the sequence of Brinkman solves at 8.4M: 43.0 and 41.8 ms;
// operator and preconditioner at 33M: 696 and 639 us.  Mixed Brinkman solves of
// other orders: lx = 6, 15.4 and 17.9 ms at 3.0M, 34.5 and 34.5 at 7.1M; lx = 4,
// 19.1 and 19.5 ms at 4.1M, 39.8 and 37.8 at 9.0M.  FP64 CG, where only the
// gather-scatter and the vector kernels are launched so, gains little above the
// line: 274 and 278 ms at 9.0M, 188 and 191 at 8.0M of lx = 5 (below, 57.7 and
// 60.3 at 2.1M); the residuals' gather-scatters 1 to 2% at most.
constexpr int64_t kDependentNodes = 6000000;
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependent_start() {
  dependent_wait();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
int launch_dependent(const ntg_plan* p, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                     A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = p->n <= kDependentNodes ? 1 : 0;
  NTG_CUDA_TRY(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...));
  NTG_COUNT_LAUNCH();
  return NTG_OK;
}

// launch helpers implemented in the .cu files
int ax_launch(ntg_plan* p, double* w, const double* u, Scalars* dot_scal, int dot_slot, cudaStream_t s);
// The direction update of the Schwarz-preconditioned CG, done by the operator
// that reads the direction: y += alpha p (the update that the iteration before
// left), p = z + beta p, then w = A p.  lx 4, 6, 8 with a dot product.
struct AxDir {
  float* p;
  const float* z;
  float* y;
  int mode;  // 0 the above; 1 start: p = z; 2 after a replacement: y is up to date
};
int ax_launch_f32(ntg_plan* p, float* w, const float* u, Scalars* dot_scal, int dot_slot, cudaStream_t s,
                  const AxDir* dir = nullptr);
int gs_launch(ntg_plan* p, double* u, int op, cudaStream_t s);
int gs_launch_f32(ntg_plan* p, float* u, int op, cudaStream_t s);
int gs_launch3(ntg_plan* p, double* u0, double* u1, double* u2, cudaStream_t s);
int gs_cls_launch3(ntg_plan* p, double* u0, double* u1, double* u2, cudaStream_t s);
int mask_launch(ntg_plan* p, double* u, cudaStream_t s);
int mask_launch_f32(ntg_plan* p, float* u, cudaStream_t s);
// assembled masked operator w = mask(gs(A u)); optional fused (u, Au_local)
int op_apply(ntg_plan* p, double* w, const double* u, cudaStream_t s);
int op_apply_f32(ntg_plan* p, float* w, const float* u, cudaStream_t s);
// generic deterministic weighted dot: sum a*b*c (c may be null -> 1)
int wdot(ntg_plan* p, const double* a, const double* b, const double* c, int64_t n, double* host_out,
         cudaStream_t s);
int gs_add_guarded(ntg_plan* p, double* u, cudaStream_t s, const Scalars* sc);
int gs_add_guarded_f32(ntg_plan* p, float* u, cudaStream_t s, const Scalars* sc);
int mask_guarded(ntg_plan* p, double* u, cudaStream_t s, const Scalars* sc);
int mask_guarded_f32(ntg_plan* p, float* u, cudaStream_t s, const Scalars* sc);
int ensure_fp32(ntg_plan* p);
int build_gs_classes(ntg_plan* p);
template <typename T>
int gs_cls_launch(ntg_plan* p, T* u, int op, cudaStream_t s, const Scalars* sc);
int grid_for(int64_t work, int threads);
int grid_red(int64_t work, int threads);
// mult (multf: after ensure_fp32) with the Dirichlet nodes' weights negative, built on first use after set_mask
int plan_multm(ntg_plan* p, const double** out);
int plan_multm(ntg_plan* p, const float** out);
int jacobi_update(ntg_plan* p);
void mask_free(ntg_mask_state* m);
// the element counts of a Schwarz preconditioner built on a structured box
// (1), or 0 for one built on a general mesh
int schwarz_box(const ntg_schwarz* w, int* ex, int* ey, int* ez);
// restarted flexible GMRES (gmres.cu)
struct GmresWork;
struct GmresOpts {
  int restart = 30, fp32 = 0, max_iter = 1000, check_every = 4;
  double rtol = 1e-10, abstol = 0.0, delta = 1e-4;
};
int gmres_solve(ntg_plan* p, GmresWork*& g, Scalars* sc, ntg_schwarz* sw, const GmresOpts& o, double* x,
                const double* f, ntg_monitor* mon);
void gmres_free(GmresWork* g);
// GLL nodes, weights and differentiation matrix of lx points
void gll_basis(int lx, double* xi, double* w, double* D);
int num_sms();
}  // namespace ntg
