// Shared pieces of the FP64 element-tile derivative kernels (deriv.cu,
// pnpn.cu): the D matrix and GLL weights as a kernel parameter, the block
// shape (elements per block for NT element tiles of shared memory), the
// reference-direction derivatives of a tile, and the launch helpers.  In fixed
// point (fx.cuh) both advection terms and the forcing of 2717 elements of
// lx = 7 take 0.46 ms where FP64 sums took 1.39.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fx.cuh"

namespace ntg {
namespace dv {

template <int LX>
struct DMat {
  double d[LX * LX];
  double w[LX];  // GLL weights
};

template <int LX, int NT>
struct Shape {
  static constexpr int LX2 = LX * LX, LX3 = LX2 * LX;
  static constexpr int EPB0 = 256 / LX2 < 1 ? 1 : 256 / LX2;
  static constexpr int EPBS = 45056 / (NT * LX3 * 8) < 1 ? 1 : 45056 / (NT * LX3 * 8);
  static constexpr int EPB = EPB0 < EPBS ? EPB0 : EPBS;
  static constexpr int NW = EPB * LX2, THREADS = (NW + 31) / 32 * 32;
};

// Blocks of the kernels whose contractions run in fixed point (fx.cuh): EPB
// elements and about one thread per line of a field's three directions.
template <int LX, int TILES>
struct FxShape {
  static constexpr int L2 = LX * LX, L3 = L2 * LX, TS = fx::Tile<LX>::SIZE;
  // elements per block: their 3 L2 lines fill the warps (100% at lx 2 and 4, 98 at 3 and 5, 96 at 6)
  static constexpr int EPB = LX <= 2 ? 16 : LX == 3 ? 7 : LX == 4 ? 4 : LX == 5 ? 5 : LX == 6 ? 2 : 1;
  // lx = 7 and 8: two whole passes over the nodes (256 against 192 threads at lx = 8: 2.50 and 2.56 ms for the
  // residuals at 24^3 elements)
  static constexpr int NT = LX == 8 ? 256 : LX == 7 ? 192 : (EPB * 3 * L2 + 31) / 32 * 32;
  // per element: tiles, the exponents of a flux's lines; once: the products of the GLL weights
  static constexpr int EL = TILES * TS + (3 * L2 + 1) / 2;
  static constexpr size_t SMEM = (size_t)(EPB * EL + L3) * sizeof(double);
  static constexpr int FIT = (int)(230000 / (SMEM + 1024)), WANT = 1344 / NT;
  static constexpr int MINB = FIT < 1 ? 1 : FIT < WANT ? FIT : WANT;
};

// the weights' products at the nodes, staged once per block
template <int LX>
__device__ __forceinline__ void stage_w3(double* w3, const DMat<LX>& M, int nt) {
  for (int t = threadIdx.x; t < LX * LX * LX; t += nt) w3[t] = M.w[t % LX] * M.w[t / LX % LX] * M.w[t / (LX * LX)];
}

template <int LX, int TILES>
int fx_grid(const ntg_plan* p) {
  using S = FxShape<LX, TILES>;
  const int64_t g = (p->nelv + S::EPB - 1) / S::EPB, cap = (int64_t)num_sms() * S::MINB;
  return (int)(g < cap ? g : cap);
}

// The kernels with these walk elements in three kinds of passes: over nodes
// (loads, metric products, results), over lines of one direction or of all
// three (derivatives, fx::deriv_line / flux_line) and barriers between.
// What bounds them is the FP64 pipe (2 operations per clock and SM), which
// only the metric products still use; the contractions run beside them on
// the integer pipes (k_vel_res, 4096 elements of lx = 8: FP64 pipe 67% of its
// rate, integer and logic 37, wide multiply-adds 13, 1.7 instructions a clock).
// NODES / LINES number the work items of a block's ne
// elements: item t -> element el of the block, node or line.
#define NTG_FX_PROLOGUE(TILES)                                                                  \
  using S = FxShape<LX, TILES>;                                                                 \
  using TL = fx::Tile<LX>;                                                                      \
  constexpr int L2 = S::L2, L3 = S::L3, TS = S::TS, EPB = S::EPB, NT = S::NT, EL = S::EL;       \
  extern __shared__ double fxs[];                                                               \
  double* w3t = fxs + EPB * EL;                                                                 \
  (void)w3t;
#define NTG_FX_ELEMENTS for (int64_t e0 = blockIdx.x * (int64_t)EPB; e0 < nelv; e0 += (int64_t)gridDim.x * EPB)
#define NTG_FX_NE const int ne = nelv - e0 < EPB ? (int)(nelv - e0) : EPB
#define NTG_FX_NODES for (int t = threadIdx.x; t < ne * L3; t += NT)
#define NTG_FX_NODE                                                                             \
  const int el = EPB == 1 ? 0 : t / L3, node = EPB == 1 ? t : t - el * L3, p = TL::at(node);    \
  const int64_t q = e0 * L3 + t;                                                                \
  double* T = fxs + el * EL;                                                                    \
  (void)p; (void)T; (void)q;
#define NTG_FX_LINES for (int t = threadIdx.x; t < ne * 3 * L2; t += NT)
#define NTG_FX_LINE                                                                             \
  const int el = EPB == 1 ? 0 : t / (3 * L2), r = EPB == 1 ? t : t - el * 3 * L2, d = r / L2;   \
  const int lq = r - d * L2;                                                                    \
  double* T = fxs + el * EL;

// reference derivatives at (i, j, k) of the tile s (s[c * LX2 + b * LX + a])
template <int LX>
__device__ __forceinline__ void rgrad(const double* s, const DMat<LX>& M, int i, int j, int k, double& ur, double& us,
                                      double& ut) {
  constexpr int LX2 = LX * LX;
  ur = us = ut = 0.0;
#pragma unroll
  for (int l = 0; l < LX; ++l) {
    ur = fma(M.d[i * LX + l], s[k * LX2 + j * LX + l], ur);
    us = fma(M.d[j * LX + l], s[k * LX2 + l * LX + i], us);
    ut = fma(M.d[k * LX + l], s[l * LX2 + j * LX + i], ut);
  }
}

template <int LX>
DMat<LX> dmat(const ntg_plan* p) {
  DMat<LX> M;
  for (int q = 0; q < LX * LX; ++q) M.d[q] = p->D[q];
  for (int q = 0; q < LX; ++q) M.w[q] = p->wq[q];
  return M;
}

template <int NT, typename F>
int dispatch(int lx, F&& f) {
  switch (lx) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 5: return f(std::integral_constant<int, 5>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 7: return f(std::integral_constant<int, 7>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 9: return f(std::integral_constant<int, 9>{});
    case 10: return f(std::integral_constant<int, 10>{});
    default: set_error("derivative operators: lx=%d not compiled (2..10)", lx); return NTG_ERR_UNSUPPORTED;
  }
}

template <int LX, int NT>
int grid_of(const ntg_plan* p) {
  constexpr int EPB = Shape<LX, NT>::EPB;
  const int64_t g = (p->nelv + EPB - 1) / EPB, cap = (int64_t)num_sms() * 32;
  return (int)(g < cap ? g : cap);
}

}  // namespace dv

inline int need_metrics(const ntg_plan* p) {
  if (!p->met) {
    set_error("derivative operators: call ntg_metrics_set(plan, x, y, z) first");
    return NTG_ERR_INVALID;
  }
  return NTG_OK;
}

// w = gs(B curl(scale u)), scale null: 1 (deriv.cu)
int curl_gs(ntg_plan* p, double* w0, double* w1, double* w2, const double* ux, const double* uy, const double* uz,
            const double* scale);

// n-double device scratch owned by the plan (grown on demand, freed with it)
double* plan_scratch(ntg_plan* p, int64_t count);

}  // namespace ntg
