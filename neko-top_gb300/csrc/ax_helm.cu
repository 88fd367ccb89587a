// Matrix-free spectral-element Helmholtz operator (ax_helm) on sm_103a:
//   w = h1 * (D^T G D) u + h2 * B * u   (element-local, unassembled)
//
// Replaces Neko's ax_helm (created by ax_helm_factory(Ax, full_formulation =
// .false.) at sources/mapping_functions/PDE_filter_mapping.f90:177 and
// sources/adjoint/adjoint_pnpn.f90:207,217; applied inside ksp%solve).
//
// The FP32 operator of the orders that have no bulk-copy pipeline (lx = 8:
// ax_helm_f32_tma.cu; FP64: ax_helm_fx.cu).  One element per LX x LX thread
// group (thread (i,j) owns the column u(i,j,0..LX-1)); EPB elements per
// block.  The t-direction contraction runs on the column held in registers
// with D taken from the kernel-parameter (constant) bank at compile-time
// indices; the r- and s-direction contractions read the element tile from
// shared memory, where a warp's reads are broadcasts or consecutive words.
// Each thread keeps its D rows/columns in registers.  The transposed
// contractions reuse the same pattern on the metric-mixed fluxes.  HBM bound
// (32 B/DOF for Poisson).
#include "common.cuh"
#include "reduce.cuh"

namespace ntg {

template <int LX>
struct DParam {
  float d[LX * LX];
};

template <int LX>
struct AxShape {
  static constexpr int LX2 = LX * LX, LX3 = LX * LX * LX;
  static constexpr int EPB_T = (256 / LX2) < 1 ? 1 : ((256 / LX2) > 8 ? 8 : 256 / LX2);
  static constexpr int EPB_S = 49152 / (3 * LX3 * (int)sizeof(float));
  static constexpr int EPB = EPB_T < EPB_S ? EPB_T : (EPB_S < 1 ? 1 : EPB_S);
  static constexpr int NW = LX2 * EPB;             // working threads
  static constexpr int NT = (NW + 31) / 32 * 32;   // launched threads
};

template <int LX, bool H1ARR, bool H2, bool DOT, bool DIR = false>
__global__ void __launch_bounds__(AxShape<LX>::NT)
    k_ax_helm(float* __restrict__ w, const float* __restrict__ u, const float* __restrict__ g11,
              const float* __restrict__ g12, const float* __restrict__ g13, const float* __restrict__ g22,
              const float* __restrict__ g23, const float* __restrict__ g33, const float* __restrict__ h1, float h1c,
              const float* __restrict__ hB, int64_t nelv, const __grid_constant__ DParam<LX> Dp, double* __restrict__ part, Scalars* sc, AxDir dir) {
  using S = AxShape<LX>;
  constexpr int LX2 = S::LX2, LX3 = S::LX3, EPB = S::EPB;
  dependent_start();
  if (DOT && sc->done) return;
  const float alpha = DIR ? (float)sc->alpha : 0.f, beta = DIR ? (float)sc->beta : 0.f;
  __shared__ float s_u[EPB][LX3];
  __shared__ float s_r[EPB][LX3];
  __shared__ float s_s[EPB][LX3];
  const int tid = threadIdx.x;
  const bool worker = tid < S::NW;
  const int le = worker ? tid / LX2 : 0;  // element slot in the block
  const int ij = worker ? tid - le * LX2 : 0;
  const int i = ij % LX, j = ij / LX;
  float Dri[LX], Dsj[LX], DTi[LX], DTj[LX];
#pragma unroll
  for (int l = 0; l < LX; ++l) {
    Dri[l] = Dp.d[i * LX + l];
    Dsj[l] = Dp.d[j * LX + l];
    DTi[l] = Dp.d[l * LX + i];
    DTj[l] = Dp.d[l * LX + j];
  }
  float dot = 0.f;  // per-thread partial in FP32 (FP64 math is scarce on GB300)
  const int64_t ngroups = (nelv + EPB - 1) / EPB;
  for (int64_t grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    const int64_t e = grp * EPB + le;
    const bool active = worker && e < nelv;
    const int64_t base = e * LX3 + ij;
    // every stream's loads first: the bytes in flight bound this kernel.  With
    // the metric loads between the contractions the operator, gather-scatter and
    // preconditioner of 4641 elements of lx = 6 took 89 us, so 81
    float ureg[LX], G[6][LX], hh[LX], zv[LX], yv[LX];
#pragma unroll
    for (int k = 0; k < LX; ++k) {
      const int64_t q = base + k * LX2;
      if constexpr (DIR) {
        ureg[k] = active && dir.mode != 1 ? dir.p[q] : 0.f;
        zv[k] = active ? dir.z[q] : 0.f;
        yv[k] = active && dir.mode == 0 ? dir.y[q] : 0.f;
      } else {
        ureg[k] = active ? u[q] : 0.f;
      }
      G[0][k] = active ? g11[q] : 0.f;
      G[1][k] = active ? g12[q] : 0.f;
      G[2][k] = active ? g13[q] : 0.f;
      G[3][k] = active ? g22[q] : 0.f;
      G[4][k] = active ? g23[q] : 0.f;
      G[5][k] = active ? g33[q] : 0.f;
      if (H1ARR) hh[k] = active ? h1[q] : 0.f;
    }
    if constexpr (DIR) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        const int64_t q = base + k * LX2;
        if (active && dir.mode == 0) dir.y[q] = yv[k] + alpha * ureg[k];
        ureg[k] = zv[k] + beta * ureg[k];
        if (active) dir.p[q] = ureg[k];
      }
    }
#pragma unroll
    for (int k = 0; k < LX; ++k)
      if (worker) s_u[le][ij + k * LX2] = ureg[k];
    __syncthreads();
    float wt[LX];
#pragma unroll
    for (int k = 0; k < LX; ++k) {
      float ur = 0.f, us = 0.f, ut = 0.f;
#pragma unroll
      for (int l = 0; l < LX; ++l) {
        ur = fma(Dri[l], s_u[le][k * LX2 + j * LX + l], ur);
        us = fma(Dsj[l], s_u[le][k * LX2 + l * LX + i], us);
        ut = fma(Dp.d[k * LX + l], ureg[l], ut);
      }
      const float h = H1ARR ? hh[k] : h1c;
      const float wr = G[0][k] * ur + G[1][k] * us + G[2][k] * ut;
      const float ws = G[1][k] * ur + G[3][k] * us + G[4][k] * ut;
      const float wtt = G[2][k] * ur + G[4][k] * us + G[5][k] * ut;
      if (worker) {
        s_r[le][ij + k * LX2] = h * wr;
        s_s[le][ij + k * LX2] = h * ws;
      }
      wt[k] = h * wtt;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LX; ++k) {
      float acc = 0.f;
#pragma unroll
      for (int l = 0; l < LX; ++l) {
        acc = fma(DTi[l], s_r[le][k * LX2 + j * LX + l], acc);
        acc = fma(DTj[l], s_s[le][k * LX2 + l * LX + i], acc);
        acc = fma(Dp.d[l * LX + k], wt[l], acc);
      }
      if (active) {
        const int64_t q = base + k * LX2;
        if (H2) acc = fma(hB[q], ureg[k], acc);
        w[q] = acc;
        if (DOT) dot = fma(ureg[k], acc, dot);
      }
    }
    // s_u is rewritten next, read last before the barrier above; s_r and s_s
    // after the next one
  }
  if (DOT) {
    double v[1] = {(double)dot};
    grid_reduce<1>(v, part, sc, FinPap());
  }
}

// TMA-pipelined FP32 kernel for lx = 8 (ax_helm_f32_tma.cu); returns
// NTG_ERR_UNSUPPORTED when a pointer is not 16-byte aligned.
int ax_f32_tma_launch(ntg_plan* p, float* w, const float* u, const float* const* g, const float* h1, float h1c,
                      const float* hB, Scalars* sc, const AxDir* dir, cudaStream_t s);

template <int LX>
static int launch_lx(ntg_plan* p, float* w, const float* u, const float* const* g, const float* h1, float h1c,
                     const float* hB, Scalars* sc, const AxDir* dir, cudaStream_t s) {
  constexpr int EPB = AxShape<LX>::EPB;
  constexpr int NT = AxShape<LX>::NT;
  DParam<LX> Dp;
  for (int q = 0; q < LX * LX; ++q) Dp.d[q] = (float)p->D[q];
  int64_t ngroups = (p->nelv + EPB - 1) / EPB;
  int64_t cap = sc ? kRedSlots : (int64_t)num_sms() * 32;
  int grid = (int)(ngroups < cap ? ngroups : cap);
  const bool h1arr = h1 != nullptr, h2 = hB != nullptr;
  const AxDir d = dir ? *dir : AxDir{};
#define NTG_AX_CASE(H1A, HH2, DT, DR)                                                                              \
  if (h1arr == H1A && h2 == HH2 && (sc != nullptr) == DT) {                                                     \
    NTG_TRY((launch_dependent(p, k_ax_helm<LX, H1A, HH2, DT, DR>, grid, NT, 0, s, w, u, g[0], g[1], g[2],    \
                              g[3], g[4], g[5], h1, h1c, hB, p->nelv, Dp, p->red_part, sc, d)));               \
  }
  if (dir) {
    // the orders of the Schwarz preconditioner
    if constexpr (LX == 4 || LX == 6 || LX == 8) {
      NTG_AX_CASE(false, false, true, true)
      NTG_AX_CASE(false, true, true, true)
      NTG_AX_CASE(true, false, true, true)
      NTG_AX_CASE(true, true, true, true)
      return NTG_OK;
    }
    set_error("ax_helm: no direction update at lx=%d", LX);
    return NTG_ERR_UNSUPPORTED;
  }
  NTG_AX_CASE(false, false, false, false)
  NTG_AX_CASE(false, true, false, false)
  NTG_AX_CASE(true, false, false, false)
  NTG_AX_CASE(true, true, false, false)
  NTG_AX_CASE(false, false, true, false)
  NTG_AX_CASE(false, true, true, false)
  NTG_AX_CASE(true, false, true, false)
  NTG_AX_CASE(true, true, true, false)
#undef NTG_AX_CASE
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

static int ax_dispatch(ntg_plan* p, float* w, const float* u, const float* const* g, const float* h1, float h1c,
                       const float* hB, Scalars* sc, const AxDir* dir, cudaStream_t s) {
  switch (p->lx) {
    case 2: return launch_lx<2>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 3: return launch_lx<3>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 4: return launch_lx<4>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 5: return launch_lx<5>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 6: return launch_lx<6>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 7: return launch_lx<7>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 8: return launch_lx<8>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 9: return launch_lx<9>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    case 10: return launch_lx<10>(p, w, u, g, h1, h1c, hB, sc, dir, s);
    default: set_error("ax_helm: lx=%d not compiled", p->lx); return NTG_ERR_UNSUPPORTED;
  }
}

int ax_launch_f32(ntg_plan* p, float* w, const float* u, Scalars* dot_scal, int, cudaStream_t s, const AxDir* dir) {
  NTG_TRY(ensure_fp32(p));
  const float* g[6] = {p->gf[0], p->gf[1], p->gf[2], p->gf[3], p->gf[4], p->gf[5]};
  timer_start(TM_AX32, s);
  const float* h1 = p->h1_const ? nullptr : p->h1f;
  const float* hB = p->ifh2 ? p->hBf : nullptr;
  int st = NTG_ERR_UNSUPPORTED;
  if (p->lx == 8 && p->use_tma) st = ax_f32_tma_launch(p, w, u, g, h1, (float)p->h1c, hB, dot_scal, dir, s);
  if (st == NTG_ERR_UNSUPPORTED) st = ax_dispatch(p, w, u, g, h1, (float)p->h1c, hB, dot_scal, dir, s);
  timer_stop(TM_AX32, s);
  return st;
}

}  // namespace ntg

using namespace ntg;

extern "C" int ntg_ax_helm(ntg_plan* plan, double* w_d, const double* u_d) {
  clear_error();
  NTG_CHECK_ARG(plan && w_d && u_d, "ntg_ax_helm: null argument");
  return ax_launch(plan, w_d, u_d, nullptr, 0, plan->stream);
}

extern "C" int ntg_ax_helm_f32(ntg_plan* plan, float* w_d, const float* u_d) {
  clear_error();
  NTG_CHECK_ARG(plan && w_d && u_d, "ntg_ax_helm_f32: null argument");
  return ax_launch_f32(plan, w_d, u_d, nullptr, 0, plan->stream);
}
