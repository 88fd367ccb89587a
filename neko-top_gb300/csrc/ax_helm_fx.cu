// The FP64 matrix-free Helmholtz operator with its contractions in fixed
// point on the integer pipes (fx.cuh).
#include <cmath>

#include "common.cuh"
#include "fx.cuh"
#include "reduce.cuh"

namespace ntg {

template <int LX>
struct FxMats {
  fx::Mat<LX, LX> D, DT;           // D and scale * D^T
  double d[LX * LX], dt[LX * LX];  // the same as FP64 numbers
};

template <int LX>
struct FxAxShape {
  static constexpr int LX2 = LX * LX, LX3 = LX2 * LX;
  static constexpr int RS = LX | 1, TILE = LX2 * RS;  // odd row stride: rows and columns without bank conflicts
  static constexpr int EPB = LX >= 7 ? 2 : LX >= 5 ? 4 : 8;
  static constexpr int NW = LX2 * EPB, NT = (NW + 31) / 32 * 32;
  static constexpr int MINB = 896 / NT;
  static constexpr size_t SMEM = EPB * (3 * TILE * sizeof(double) + 2 * LX2 * sizeof(int));
};

template <int LX, bool DOT>
__global__ void __launch_bounds__(FxAxShape<LX>::NT, FxAxShape<LX>::MINB)
    k_ax_fx(double* __restrict__ w, const double* __restrict__ u, const double* __restrict__ g11,
            const double* __restrict__ g12, const double* __restrict__ g13, const double* __restrict__ g22,
            const double* __restrict__ g23, const double* __restrict__ g33, const double* __restrict__ h1,
            const double* __restrict__ hB, int64_t nelv, const __grid_constant__ FxMats<LX> P,
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
  auto sync = [&]() {
    if constexpr (LX == 8) asm volatile("bar.sync %0, 64;" ::"r"(le + 1) : "memory");
    else __syncthreads();
  };
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
    sync();
    if (worker) {
      double x[LX];
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = U[ro + l];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, [&](int A, double y) { R[ro + A] = y; });
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = U[so + l * RS];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, [&](int A, double y) { V[so + A * RS] = y; });
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = wt[l];
      fx::line_dbl<LX, LX, true>(P.D, P.d, x, [&](int A, double y) { wt[A] = y; });
    }
    sync();
    if (act) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        const int64_t q = base + k * LX2;
        const int p = to + k * LX * RS;
        const double ur = R[p], us = V[p], ut = wt[k];
        const double a12 = g12[q], a13 = g13[q], a23 = g23[q];
        double fr = g11[q] * ur + a12 * us + a13 * ut;
        double fs = a12 * ur + g22[q] * us + a23 * ut;
        double ft = a13 * ur + a23 * us + g33[q] * ut;
        if (h1) {
          const double hh = h1[q];
          fr *= hh;
          fs *= hh;
          ft *= hh;
        }
        R[p] = fr;
        V[p] = fs;
        wt[k] = ft;
      }
    }
    sync();
    int64_t Y[LX];
    int kt = fx::kZero;
    if (worker) {
      double x[LX];
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = R[ro + l];
      kr[ab] = fx::line_int<LX, LX, true>(P.DT, P.dt, x,
                                          [&](int A, int64_t y) { R[ro + A] = __longlong_as_double(y); });
#pragma unroll
      for (int l = 0; l < LX; ++l) x[l] = V[so + l * RS];
      ks[ab] = fx::line_int<LX, LX, true>(P.DT, P.dt, x,
                                          [&](int A, int64_t y) { V[so + A * RS] = __longlong_as_double(y); });
      kt = fx::line_int<LX, LX, true>(P.DT, P.dt, wt, [&](int A, int64_t y) { Y[A] = y; });
    }
    sync();
    if (act) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        const int64_t q = base + k * LX2;
        const int p = to + k * LX * RS;
        double acc = fx::sum3(__double_as_longlong(R[p]), kr[b + LX * k], __double_as_longlong(V[p]), ks[a + LX * k],
                              Y[k], kt);
        if (DOT || hB) {
          const double uk = U[p];
          if (hB) acc = fma(hB[q], uk, acc);
          if (DOT) dot = fma(uk, acc, dot);
        }
        w[q] = acc;
      }
    }
  }
  if (DOT) {
    double v[1] = {dot};
    grid_reduce<1>(v, part, sc, FinPap());
  }
}

template <int LX>
static int launch_fx(ntg_plan* p, double* w, const double* u, const double* const* g, const double* h1, double h1c,
                     const double* hB, Scalars* sc, cudaStream_t s) {
  using S = FxAxShape<LX>;
  FxMats<LX> P;
  for (int i = 0; i < LX; ++i)
    for (int j = 0; j < LX; ++j) {
      P.d[i * LX + j] = p->D[i * LX + j];
      P.dt[i * LX + j] = p->D[j * LX + i] * (h1 ? 1.0 : h1c);
    }
  double dt[LX * LX];
  for (int i = 0; i < LX; ++i)
    for (int j = 0; j < LX; ++j) dt[i * LX + j] = p->D[j * LX + i];
  P.D = fx::make_mat<LX, LX>(p->D);
  P.DT = fx::make_mat<LX, LX>(dt, h1 ? 1.0 : h1c);
  const int64_t ngroups = (p->nelv + S::EPB - 1) / S::EPB, cap = sc ? kRedSlots : (int64_t)1 << 30;
  const int grid = (int)(ngroups < cap ? ngroups : cap);
  auto run = [&](auto kernel) -> int {
    NTG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    kernel<<<grid, S::NT, S::SMEM, s>>>(w, u, g[0], g[1], g[2], g[3], g[4], g[5], h1, hB, p->nelv, P, p->red_part, sc);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  };
  NTG_TRY(sc ? run(k_ax_fx<LX, true>) : run(k_ax_fx<LX, false>));
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

int ax_fx_launch(ntg_plan* p, double* w, const double* u, const double* const* g, const double* h1, double h1c,
                 const double* hB, Scalars* sc, cudaStream_t s) {
  // a constant h1 is folded into D^T, whose exponent offset must stay small
  if (!h1 && h1c != 0.0 && !(std::fabs(h1c) > 1e-6 && std::fabs(h1c) < 1e6)) return NTG_ERR_UNSUPPORTED;
  switch (p->lx) {
    case 4: return launch_fx<4>(p, w, u, g, h1, h1c, hB, sc, s);
    case 5: return launch_fx<5>(p, w, u, g, h1, h1c, hB, sc, s);
    case 6: return launch_fx<6>(p, w, u, g, h1, h1c, hB, sc, s);
    case 7: return launch_fx<7>(p, w, u, g, h1, h1c, hB, sc, s);
    case 8: return launch_fx<8>(p, w, u, g, h1, h1c, hB, sc, s);
    case 9: return launch_fx<9>(p, w, u, g, h1, h1c, hB, sc, s);
    case 10: return launch_fx<10>(p, w, u, g, h1, h1c, hB, sc, s);
    default: return NTG_ERR_UNSUPPORTED;
  }
}

}  // namespace ntg
