// The FP64 matrix-free Helmholtz operator with its contractions in fixed
// point on the integer pipes (fx.cuh).  With every product on the FP64 pipe it
// took 28 clocks per node and SM, 1.9 ms at 16.8M nodes of lx = 8; here it has
// the 11 operations of the metric products and the mass term, 5.5 clocks, and
// still bounds it: 0.38 ms are 7.1 clocks, against 0.18 ms for its 72 B per node
// (counters at 2.1M nodes: FP64 pipe 64%, integer and logic 40, wide
// multiply-adds 13, load/store 12, 1.7 instructions a clock and SM).  One
// element per block at lx = 8: up to sixteen blocks per SM keep the phases of
// different elements apart.
#include <cmath>

#include "common.cuh"
#include "fx.cuh"
#include "reduce.cuh"

namespace ntg {

template <int LX>
struct FxAxShape {
  static constexpr int LX2 = LX * LX, LX3 = LX2 * LX;
  static constexpr int RS = LX | 1, TILE = LX2 * RS;  // odd row stride: rows and columns without bank conflicts
  // elements per block: their lines fill the warps (98% at lx 3, 5 and 6, 96 at 7, 95 at 9, 94 at 10)
  static constexpr int EPB = LX == 8 ? 1 : LX <= 3 ? 14 : LX == 4 ? 4 : LX == 6 ? 7 : LX <= 7 ? 5 : 3;
  static constexpr int NW = LX2 * EPB, NT = (NW + 31) / 32 * 32;
  static constexpr int MINB = LX == 8 ? 16 : 896 / NT;
  static constexpr size_t SMEM = EPB * (3 * TILE * sizeof(double) + 2 * LX2 * sizeof(int));
};

// FIELD: h1 is a field (the fluxes' guard, fx::flux_line); null otherwise.  The
// pointer is tested all the same: products by h1s alone would be predicated.
// 16.8M nodes of lx = 8: constant h1 368 us; a smooth field 484 (444 without the
// guard), one that jumps between 1e-3 and 1 from node to node 660, where FP64
// sums throughout took 1979.
template <int LX, bool FIELD, bool DOT>
__global__ void __launch_bounds__(FxAxShape<LX>::NT, FxAxShape<LX>::MINB)
    k_ax_fx(double* __restrict__ w, const double* __restrict__ u, const double* __restrict__ g11,
            const double* __restrict__ g12, const double* __restrict__ g13, const double* __restrict__ g22,
            const double* __restrict__ g23, const double* __restrict__ g33, const double* __restrict__ h1,
            double h1s, const double* __restrict__ hB, int64_t nelv, const __grid_constant__ fx::Mats<LX> P,
            double* __restrict__ part, Scalars* sc) {
  using S = FxAxShape<LX>;
  constexpr int LX2 = S::LX2, LX3 = S::LX3, EPB = S::EPB, RS = S::RS, TILE = S::TILE;
  if (DOT && sc->done) return;
  extern __shared__ double fsm[];
  const int tid = threadIdx.x;
  const bool worker = tid < S::NW;
  const int le = worker ? tid / LX2 : 0, ab = worker ? tid - le * LX2 : 0, a = ab % LX, b = ab / LX;
  double* U = fsm + le * 3 * TILE;
  double* R = U + TILE;
  double* V = R + TILE;
  int* kr = reinterpret_cast<int*>(fsm + EPB * 3 * TILE) + le * 2 * LX2;
  int* ks = kr + LX2;
  const int ro = (a + LX * b) * RS;  // row (j, k) = (a, b)
  const int so = LX * b * RS + a;    // column along j at (i, k) = (a, b)
  const int to = b * RS + a;         // column along k at (i, j) = (a, b)
  double dot = 0.0;
  for (int64_t grp = blockIdx.x; grp * EPB < nelv; grp += gridDim.x) {
    const int64_t e = grp * EPB + le;
    const bool act = worker && e < nelv;
    const int64_t base = e * LX3 + ab;
    double wt[LX];  // the column: u, then its derivative, then its flux
    if (worker) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        wt[k] = act ? u[base + k * LX2] : 0.0;
        U[to + k * LX * RS] = wt[k];
      }
    }
    __syncthreads();
    if (worker) {
      double x[LX];
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = U[ro + l];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, false, [&](int A, double y) { R[ro + A] = y; });
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = U[so + l * RS];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, false, [&](int A, double y) { V[so + A * RS] = y; });
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = wt[l];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, false, [&](int A, double y) { wt[A] = y; });
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        const int64_t q = base + k * LX2;
        const int p = to + k * LX * RS;
        const double ur = R[p], us = V[p], ut = wt[k];
        const double a12 = g12[q], a13 = g13[q], a23 = g23[q];
        R[p] = g11[q] * ur + a12 * us + a13 * ut;
        V[p] = a12 * ur + g22[q] * us + a23 * ut;
        wt[k] = a13 * ur + a23 * us + g33[q] * ut;
      }
      if (h1 || h1s != 1.0) {  // its own loop: a predicated-off FP64 product takes the pipe all the same
#pragma unroll
        for (int k = 0; k < LX; ++k) {
          const int p = to + k * LX * RS;
          const double hh = h1 ? h1[base + k * LX2] : h1s;
          R[p] *= hh;
          V[p] *= hh;
          wt[k] *= hh;
        }
      }
    }
    __syncthreads();
    int64_t Y[LX];
    int kt = fx::kZero;
    if (worker) {
      double x[LX];
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = R[ro + l];
      kr[ab] = fx::line_int_to<LX, LX, true>(P.DT, P.dt, x, FIELD, R + ro, 1);
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = V[so + l * RS];
      ks[ab] = fx::line_int_to<LX, LX, true>(P.DT, P.dt, x, FIELD, V + so, RS);
      kt = fx::line_int<LX, LX, true>(
          P.DT, P.dt, wt, FIELD, [&](int A, int64_t y) { Y[A] = y; }, [&](int A) { return Y[A]; });
    }
    __syncthreads();
    if (act) {
      double acc[LX];
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        const int p = to + k * LX * RS;
        acc[k] = fx::sum3(__double_as_longlong(R[p]), kr[b + LX * k], __double_as_longlong(V[p]), ks[a + LX * k],
                          Y[k], kt);
      }
      if (hB) {
#pragma unroll
        for (int k = 0; k < LX; ++k) acc[k] = fma(hB[base + k * LX2], U[to + k * LX * RS], acc[k]);
      }
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        w[base + k * LX2] = acc[k];
        if (DOT) dot = fma(U[to + k * LX * RS], acc[k], dot);
      }
    }
  }
  if (DOT) {
    double v[1] = {dot};
    grid_reduce<1>(v, part, sc, FinPap());
  }
}

template <int LX, bool FIELD, bool DOT>
static int launch_fx(ntg_plan* p, double* w, const double* u, const double* const* g, const double* h1, double h1c,
                     const double* hB, Scalars* sc, cudaStream_t s) {
  using S = FxAxShape<LX>;
  const double fold = !FIELD && fx::foldable(h1c) ? h1c : 1.0;  // a constant h1 goes into D^T
  const double h1s = FIELD || fold == h1c ? 1.0 : h1c;
  const fx::Mats<LX> P = fx::plan_mats<LX>(p, fold);
  const int64_t ngroups = (p->nelv + S::EPB - 1) / S::EPB, cap = DOT ? kRedSlots : (int64_t)1 << 30;
  const int grid = (int)(ngroups < cap ? ngroups : cap);
  NTG_TRY((fx::use_smem<k_ax_fx<LX, FIELD, DOT>>(S::SMEM)));
  k_ax_fx<LX, FIELD, DOT><<<grid, S::NT, S::SMEM, s>>>(w, u, g[0], g[1], g[2], g[3], g[4], g[5], h1, h1s, hB, p->nelv, P,
                                                    p->red_part, sc);
  NTG_COUNT_LAUNCH();
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

template <int LX>
static int launch_fx(ntg_plan* p, double* w, const double* u, const double* const* g, const double* h1, double h1c,
                     const double* hB, Scalars* sc, cudaStream_t s) {
  if (h1) return sc ? launch_fx<LX, true, true>(p, w, u, g, h1, h1c, hB, sc, s)
                    : launch_fx<LX, true, false>(p, w, u, g, h1, h1c, hB, sc, s);
  return sc ? launch_fx<LX, false, true>(p, w, u, g, h1, h1c, hB, sc, s)
            : launch_fx<LX, false, false>(p, w, u, g, h1, h1c, hB, sc, s);
}

int ax_launch(ntg_plan* p, double* w, const double* u, Scalars* dot_scal, int, cudaStream_t s) {
  const double* g[6] = {p->g[0], p->g[1], p->g[2], p->g[3], p->g[4], p->g[5]};
  const double* h1 = p->h1_const ? nullptr : p->h1;
  const double* hB = p->ifh2 ? p->hB : nullptr;
  timer_start(TM_AX64, s);
  int st = NTG_OK;
  switch (p->lx) {
    case 2: st = launch_fx<2>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 3: st = launch_fx<3>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 4: st = launch_fx<4>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 5: st = launch_fx<5>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 6: st = launch_fx<6>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 7: st = launch_fx<7>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 8: st = launch_fx<8>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 9: st = launch_fx<9>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    case 10: st = launch_fx<10>(p, w, u, g, h1, p->h1c, hB, dot_scal, s); break;
    default: set_error("ax_helm: lx=%d not compiled", p->lx); st = NTG_ERR_UNSUPPORTED;
  }
  timer_stop(TM_AX64, s);
  return st;
}

}  // namespace ntg
