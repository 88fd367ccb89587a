// Dealiased (over-integrated) adjoint and linearised advection, FP64
// (sources/adjoint/adv_adjoint_dealias.f90: init_dealias :137-224,
// compute_adjoint_advection_dealias :235-462, compute_linear_advection_dealias
// :470-600).  The fields are interpolated from the LX GLL points to LXD
// Gauss-Legendre points per direction (J), the products are formed there with
// the GL weights and the metric cofactors interpolated to GL, and the result
// comes back with J^T:
//
//   adjoint  f_i -= J^T [ sum_j u_j opgrad_i(Ub_j) + sum_d cdtp_d(u_i Ub_d) ]
//   linear   f_i -= J^T [ u . opgrad(Ub_i) + Ub . opgrad(u_i) ]
//
// The reference round-trips the interpolated fields, their derivatives and
// the fluxes through device arrays (20 GL-sized scratch fields); here only
// the GL cofactors (9 doubles per GL point, interpolated once at create)
// stream from memory.  The sums are rewritten with contravariant velocities,
// so the three cdtp of a component become one transposed derivative and the
// linear term needs none.  The contractions run in fixed point (fx.cuh): the
// adjoint term of 24^3 elements, lx = 8, takes 5.3 ms where FP64 sums took
// 22.5, the linear one of 315 elements, lx = 6, 63 us where they took 201.
// Latency bounds it: the tiles of LXD^3 64-bit values leave room for 14 warps per
// SM at lx = 8, with some 20 barriers per element, and these issue 1.3
// instructions per clock and SM, 2,960 per GL point (counters at 4096 elements:
// integer and logic pipe 31% of its rate, FP64 29, wide multiply-adds 12,
// load/store 6).
#include <cmath>

#include "deriv.cuh"

struct ntg_dealias {
  ntg_plan* p = nullptr;
  int lx = 0, lxd = 0;
  int64_t ngl = 0;  // nelv * lxd^3
  double J[16 * NTG_LXMAX];
  double Dg[16 * 16];
  double wg[16];
  double* met_gl = nullptr;  // 9 x ngl cofactors at the GL points
  int grid = 0;
  size_t smem = 0;
  std::shared_ptr<void> mats;  // the fixed-point matrices of the advection kernels
};

namespace ntg {
namespace dl {

constexpr int NT = 256;

template <int LX, int LXD>
struct GLMat {
  double J[LXD * LX];  // J[A * LX + a] = l_a(xg_A)
};

template <int LX, int LXD>
struct Smem {
  static constexpr int N3 = LXD * LXD * LXD, TA = LXD * LX * LX, TB = LXD * LXD * LX, G3 = LX * LX * LX;
  static constexpr int DOUBLES = 2 * N3 + TA + TB + LXD * LX;
  static constexpr size_t BYTES = sizeof(double) * DOUBLES;
};

// dst[C][B][A] = sum J[C][c] J[B][b] J[A][a] src[c][b][a] (block-cooperative)
template <int LX, int LXD>
__device__ __forceinline__ void to_gl(double* dst, const double* src, double* tA, double* tB, const double* J) {
  for (int t = threadIdx.x; t < LX * LX * LXD; t += NT) {
    const int A = t % LXD, cb = t / LXD;
    double acc = 0.0;
#pragma unroll
    for (int a = 0; a < LX; ++a) acc = fma(J[A * LX + a], src[cb * LX + a], acc);
    tA[t] = acc;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < LX * LXD * LXD; t += NT) {
    const int A = t % LXD, B = (t / LXD) % LXD, c = t / (LXD * LXD);
    double acc = 0.0;
#pragma unroll
    for (int b = 0; b < LX; ++b) acc = fma(J[B * LX + b], tA[(c * LX + b) * LXD + A], acc);
    tB[t] = acc;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < LXD * LXD * LXD; t += NT) {
    const int BA = t % (LXD * LXD), C = t / (LXD * LXD);
    double acc = 0.0;
#pragma unroll
    for (int c = 0; c < LX; ++c) acc = fma(J[C * LX + c], tB[c * LXD * LXD + BA], acc);
    dst[t] = acc;
  }
  __syncthreads();
}

// out[c][b][a] (+)= sign * sum J[C][c] J[B][b] J[A][a] src[C][B][A]; out in global memory
template <int LX, int LXD>
__device__ __forceinline__ void to_gll(double* __restrict__ out, const double* src, double* tA, double* tB,
                                       const double* J) {
  for (int t = threadIdx.x; t < LX * LXD * LXD; t += NT) {
    const int BA = t % (LXD * LXD), c = t / (LXD * LXD);
    double acc = 0.0;
#pragma unroll
    for (int C = 0; C < LXD; ++C) acc = fma(J[C * LX + c], src[C * LXD * LXD + BA], acc);
    tB[t] = acc;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < LX * LX * LXD; t += NT) {
    const int A = t % LXD, b = (t / LXD) % LX, c = t / (LXD * LX);
    double acc = 0.0;
#pragma unroll
    for (int B = 0; B < LXD; ++B) acc = fma(J[B * LX + b], tB[(c * LXD + B) * LXD + A], acc);
    tA[t] = acc;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < LX * LX * LX; t += NT) {
    const int a = t % LX, cb = t / LX;
    double acc = 0.0;
#pragma unroll
    for (int A = 0; A < LXD; ++A) acc = fma(J[A * LX + a], tA[cb * LXD + A], acc);
    out[t] = acc;
  }
  __syncthreads();
}

// out = to_gl(in) (DIR 0) or to_gll(in) (DIR 1) for `nf` fields (stride = field size)
template <int LX, int LXD, int DIR>
__global__ void __launch_bounds__(NT) k_map(double* __restrict__ out, const double* __restrict__ in, int nf,
                                            int64_t nelv, int64_t n_in, int64_t n_out,
                                            const __grid_constant__ GLMat<LX, LXD> M) {
  using S = Smem<LX, LXD>;
  extern __shared__ double sm[];
  double* tile = sm;
  double* tA = sm + 2 * S::N3;
  double* tB = tA + S::TA;
  double* J = tB + S::TB;
  for (int t = threadIdx.x; t < LXD * LX; t += NT) J[t] = M.J[t];
  constexpr int NIN = DIR == 0 ? S::G3 : S::N3;
  constexpr int NOUT = DIR == 0 ? S::N3 : S::G3;
  __syncthreads();
  for (int64_t e = blockIdx.x; e < nelv; e += gridDim.x) {
    for (int f = 0; f < nf; ++f) {
      const double* src = in + f * n_in + e * NIN;
      double* dst = out + f * n_out + e * NOUT;
      for (int t = threadIdx.x; t < NIN; t += NT) tile[t] = src[t];
      __syncthreads();
      if (DIR == 0) {
        to_gl<LX, LXD>(tile + S::N3, tile, tA, tB, J);
        for (int t = threadIdx.x; t < S::N3; t += NT) dst[t] = tile[S::N3 + t];
      } else {
        to_gll<LX, LXD>(dst, tile, tA, tB, J);
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// The advection terms.  Everything between the GLL loads and the GLL update
// stays in shared memory (12 tiles of LXD^3 numbers); the contractions (nine
// interpolations, the GL derivatives and their transposes) run in fixed
// point on the integer pipes (fx.cuh), the products on the FP64 pipe.
//
// The GL weights never appear in a product: they are folded into the
// interpolation back (JW = J^T W per direction), which leaves the transposed
// derivative acting before them, DT = W^-1 D^T W.  With V_d = sum_c c_dc
// Ub_c and a_d = sum_j u_j dUb_j/dr_d the adjoint term of component i is
//   sum_d c_di a_d + sum_d DT_d (u_i V_d)
// (39 FP64 operations per GL point where mixing each gradient first and
// weighting each product takes 162 with the contractions), the linear one
//   sum_d (V_d(u) dUb_i/dr_d + V_d(Ub) du_i/dr_d)     (36).
// ---------------------------------------------------------------------------
template <int LX, int LXD>
struct AdvMats {
  fx::Mat<LX, LXD> J;
  fx::Mat<LXD, LX> JW;
  fx::Mat<LXD, LXD> D, DT;
  double j[LXD * LX], jw[LX * LXD], d[LXD * LXD], dt[LXD * LXD];
};

template <int LX, int LXD>
struct AdvShape {
  using TG = fx::Tile<LXD>;
  static constexpr int G2 = LXD * LXD, G3 = G2 * LXD, L2 = LX * LX, L3 = L2 * LX, RS = TG::RS, TS = TG::SIZE;
  // elements per block: nearly whole warps (432 of 448 threads at lxd 6, 441 of 448 at 7)
  static constexpr int EPB = LXD == 6 ? 4 : LXD == 7 ? 3 : 1;
  static constexpr int NT = (EPB * 3 * G2 + 31) / 32 * 32;  // a thread per line of three fields or directions
  static constexpr int EL = 12 * TS + (3 * G2 + 1) / 2;     // doubles per element: tiles, line exponents
  static constexpr size_t SMEM = sizeof(double) * EPB * EL;
  static constexpr int MINB = (int)(232448 / (SMEM + 1024));
  // the interpolations' intermediate forms fit the tiles they pass through
  static_assert(L2 * (LX | 1) * 6 <= 6 * TS && L2 * RS * 6 <= 6 * TS && LX * LXD * RS * 6 <= 6 * TS, "tiles");
};

template <int NIN, int NOUT, bool ANTI>
__device__ __forceinline__ void line_at(const fx::Mat<NIN, NOUT>& M, const double* Md, const double* in, int si,
                                        double* out, int so) {
  double x[NIN];
#pragma unroll
  for (int l = 0; l < NIN; ++l) x[l] = in[l * si];
  fx::line_dbl<NIN, NOUT, ANTI>(M, Md, x, false, [&](int A, double y) { out[A * so] = y; });
}

// MODE 0: adjoint, MODE 1: linear
template <int LX, int LXD, int MODE>
__global__ void __launch_bounds__(AdvShape<LX, LXD>::NT, AdvShape<LX, LXD>::MINB)
    k_adv(double* __restrict__ f0, double* __restrict__ f1, double* __restrict__ f2, const double* __restrict__ u0,
          const double* __restrict__ u1, const double* __restrict__ u2, const double* __restrict__ b0,
          const double* __restrict__ b1, const double* __restrict__ b2, const double* __restrict__ met, int64_t ngl,
          int64_t nelv, const __grid_constant__ AdvMats<LX, LXD> P) {
  using S = AdvShape<LX, LXD>;
  using TG = fx::Tile<LXD>;
  constexpr int G2 = S::G2, G3 = S::G3, L2 = S::L2, L3 = S::L3, RS = S::RS, TS = S::TS, EPB = S::EPB, NT = S::NT;
  constexpr int LS = LX | 1, RES = MODE == 0 ? 9 : 6;  // first tile of the results
  extern __shared__ double sm[];
  for (int64_t e0 = blockIdx.x * (int64_t)EPB; e0 < nelv; e0 += (int64_t)gridDim.x * EPB) {
    const int ne = nelv - e0 < EPB ? (int)(nelv - e0) : EPB;
    // items t of `per` per element: element slot, index in it
    auto items = [&](int per, auto&& fn) {
      for (int t = threadIdx.x; t < ne * per; t += NT) {
        const int el = EPB == 1 ? 0 : t / per;
        fn(sm + el * S::EL, EPB == 1 ? t : t - el * per, e0 + el);
      }
    };
    // the fields (u, Ub), staged by rows of LS; J along r, s, t
    items(6 * L3, [&](double* T, int i, int64_t e) {
      const int f = i / L3, node = i - f * L3;
      const double* src = f == 0 ? u0 : f == 1 ? u1 : f == 2 ? u2 : f == 3 ? b0 : f == 4 ? b1 : b2;
      T[6 * TS + (f * L2 + node / LX) * LS + node % LX] = src[e * L3 + node];
    });
    __syncthreads();
    items(6 * L2, [&](double* T, int i, int64_t) {
      line_at<LX, LXD, false>(P.J, P.j, T + 6 * TS + i * LS, 1, T + i * RS, 1);
    });
    __syncthreads();
    items(6 * LX * LXD, [&](double* T, int i, int64_t) {  // (f, c), A
      const int fc = i / LXD, A = i - fc * LXD;
      line_at<LX, LXD, false>(P.J, P.j, T + fc * LX * RS + A, RS, T + 6 * TS + fc * LXD * RS + A, RS);
    });
    __syncthreads();
    items(6 * G2, [&](double* T, int i, int64_t) {  // f, B, A
      const int f = i / G2, r = i - f * G2, p = r / LXD * RS + r % LXD;
      line_at<LX, LXD, false>(P.J, P.j, T + 6 * TS + f * LX * LXD * RS + p, LXD * RS, T + f * TS + p, LXD * RS);
    });
    __syncthreads();
    // tiles 0-2: u, 3-5: Ub; adjoint: 6-8 fluxes, 9-11 a_d, then the result per
    // component; linear: 6-8 the result, 9-11 V_d of the undifferentiated field
    if constexpr (MODE == 0) {
      // a_d along its lines: the three fields' derivatives of one line each
      // are weighted by u and summed in registers
      items(3 * G2, [&](double* T, int t, int64_t) {
        const int d = t / G2, b = TG::base(d, t - d * G2), st = TG::stride(d);
        double a[LXD];
#pragma unroll
        for (int l = 0; l < LXD; ++l) a[l] = 0.0;
#pragma unroll 1
        for (int f = 0; f < 3; ++f) {
          const double *u = T + f * TS + b, *v = T + (3 + f) * TS + b;
          double x[LXD];
#pragma unroll
          for (int l = 0; l < LXD; ++l) x[l] = v[l * st];
          fx::line_dbl<LXD, LXD, true>(P.D, P.d, x, false, [&](int A, double y) { a[A] = fma(y, u[A * st], a[A]); });
        }
        double* o = T + (9 + d) * TS + b;
#pragma unroll
        for (int l = 0; l < LXD; ++l) o[l * st] = a[l];
      });
      __syncthreads();
      items(G3, [&](double* T, int node, int64_t e) {
        const int p = TG::at(node);
        const int64_t q = e * G3 + node;
        double c[9];
#pragma unroll
        for (int m = 0; m < 9; ++m) c[m] = met[m * ngl + q];
        const double vx = T[3 * TS + p], vy = T[4 * TS + p], vz = T[5 * TS + p];
        const double ar = T[9 * TS + p], as = T[10 * TS + p], at = T[11 * TS + p];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          T[(3 + m) * TS + p] = c[3 * m] * vx + c[3 * m + 1] * vy + c[3 * m + 2] * vz;
          T[(9 + m) * TS + p] = c[m] * ar + c[3 + m] * as + c[6 + m] * at;
        }
      });
      __syncthreads();
#pragma unroll 1
      for (int i = 0; i < 3; ++i) {
        items(3 * G2, [&](double* T, int t, int64_t) {
          const int d = t / G2, b = TG::base(d, t - d * G2), st = TG::stride(d);
          const double *u = T + i * TS + b, *v = T + (3 + d) * TS + b;
          double* o = T + (6 + d) * TS + b;
          double x[LXD];
#pragma unroll
          for (int l = 0; l < LXD; ++l) x[l] = u[l * st] * v[l * st];
          reinterpret_cast<int*>(T + 12 * TS)[t] = fx::line_int_to<LXD, LXD, true>(P.DT, P.dt, x, false, o, st);
        });
        __syncthreads();
        items(G3, [&](double* T, int node, int64_t) {
          const int p = TG::at(node);
          T[(9 + i) * TS + p] += fx::flux_sum<LXD>(T + 6 * TS, T + 7 * TS, T + 8 * TS,
                                                   reinterpret_cast<const int*>(T + 12 * TS), node);
        });
        __syncthreads();
      }
    } else {
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        items(G3, [&](double* T, int node, int64_t e) {
          const int p = TG::at(node);
          const int64_t q = e * G3 + node;
          const double* X = T + (pass ? 3 : 0) * TS + p;
          const double x = X[0], y = X[TS], z = X[2 * TS];
          if (pass == 0) T[6 * TS + p] = T[7 * TS + p] = T[8 * TS + p] = 0.0;
#pragma unroll
          for (int m = 0; m < 3; ++m)
            T[(9 + m) * TS + p] = met[3 * m * ngl + q] * x + met[(3 * m + 1) * ngl + q] * y + met[(3 * m + 2) * ngl + q] * z;
        });
        __syncthreads();
        // the sums of tiles 6-8 line by line, one direction at a time
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
          items(3 * G2, [&](double* T, int t, int64_t) {
            const int i = t / G2, b = TG::base(d, t - i * G2), st = TG::stride(d);
            const double *in = T + ((pass ? 0 : 3) + i) * TS + b, *v = T + (9 + d) * TS + b;
            double* o = T + (6 + i) * TS + b;
            double x[LXD];
#pragma unroll
            for (int l = 0; l < LXD; ++l) x[l] = in[l * st];
            fx::line_dbl<LXD, LXD, true>(P.D, P.d, x, false, [&](int A, double y) {
              o[A * st] = fma(y, v[A * st], o[A * st]);
            });
          });
          __syncthreads();
        }
      }
    }
    // back: JW along t, s, r, then f -= the result
    items(3 * G2, [&](double* T, int t, int64_t) {  // i, B, A
      const int i = t / G2, r = t - i * G2, p = r / LXD * RS + r % LXD;
      line_at<LXD, LX, false>(P.JW, P.jw, T + (RES + i) * TS + p, LXD * RS, T + i * LX * LXD * RS + p, LXD * RS);
    });
    __syncthreads();
    items(3 * LX * LXD, [&](double* T, int t, int64_t) {  // (i, c), A
      const int ic = t / LXD, A = t - ic * LXD;
      line_at<LXD, LX, false>(P.JW, P.jw, T + ic * LXD * RS + A, RS, T + 6 * TS + ic * LX * RS + A, RS);
    });
    __syncthreads();
    items(3 * L2, [&](double* T, int t, int64_t) {  // (i, c, b)
      line_at<LXD, LX, false>(P.JW, P.jw, T + 6 * TS + t * RS, 1, T + t * LS, 1);
    });
    __syncthreads();
    items(3 * L3, [&](double* T, int t, int64_t e) {
      const int i = t / L3, node = t - i * L3;
      double* f = (i == 0 ? f0 : i == 1 ? f1 : f2) + e * L3 + node;
      *f -= T[(i * L2 + node / LX) * LS + node % LX];
    });
    // the next element's fields go to tiles 6 on, read last before the barrier above
  }
}

template <int LX, int LXD>
AdvMats<LX, LXD> adv_mats(const ntg_dealias* d) {
  AdvMats<LX, LXD> P;
  long double dt[LXD * LXD];
  for (int A = 0; A < LXD; ++A) {
    for (int a = 0; a < LX; ++a) {
      P.j[A * LX + a] = d->J[A * LX + a];
      P.jw[a * LXD + A] = d->J[A * LX + a] * d->wg[A];
    }
    for (int l = 0; l < LXD; ++l) {
      P.d[A * LXD + l] = d->Dg[A * LXD + l];
      dt[A * LXD + l] = (long double)d->Dg[l * LXD + A] * d->wg[l] / d->wg[A];
      P.dt[A * LXD + l] = (double)dt[A * LXD + l];
    }
  }
  P.J = fx::make_mat<LX, LXD>(d->J);
  long double jw[LX * LXD];
  for (int a = 0; a < LX; ++a)
    for (int A = 0; A < LXD; ++A) jw[a * LXD + A] = (long double)d->J[A * LX + a] * d->wg[A];
  P.JW = fx::make_mat<LXD, LX>(jw);
  P.D = fx::make_mat<LXD, LXD>(d->Dg);
  P.DT = fx::make_mat<LXD, LXD>(dt);
  return P;
}

template <int LX, int LXD>
GLMat<LX, LXD> glmat(const ntg_dealias* d) {
  GLMat<LX, LXD> M;
  for (int q = 0; q < LXD * LX; ++q) M.J[q] = d->J[q];
  return M;
}

template <typename F>
int dispatch(int lx, int lxd, F&& f) {
  if (lx == 4 && lxd == 6) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 6>{});
  if (lx == 5 && lxd == 7) return f(std::integral_constant<int, 5>{}, std::integral_constant<int, 7>{});
  if (lx == 6 && lxd == 9) return f(std::integral_constant<int, 6>{}, std::integral_constant<int, 9>{});
  if (lx == 7 && lxd == 10) return f(std::integral_constant<int, 7>{}, std::integral_constant<int, 10>{});
  if (lx == 8 && lxd == 12) return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 12>{});
  set_error("dealiasing: (lx, lxd) = (%d, %d) not compiled; pairs: (4,6) (5,7) (6,9) (7,10) (8,12)", lx, lxd);
  return NTG_ERR_UNSUPPORTED;
}

// Gauss-Legendre points and weights (Newton on the three-term recurrence of
// P_n from the Chebyshev-like start cos(pi (i + 3/4) / (n + 1/2)))
void gauss_legendre(int n, double* x, double* w) {
  for (int i = 0; i < n; ++i) {
    double z = cos(M_PI * (i + 0.75) / (n + 0.5)), dp = 1.0;
    for (int it = 0; it < 100; ++it) {
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; ++k) {
        const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = n * (z * p1 - p0) / (z * z - 1.0);
      const double dz = p1 / dp;
      z -= dz;
      if (fabs(dz) < 1e-16) break;
    }
    double p0 = 1.0, p1 = z;
    for (int k = 2; k <= n; ++k) {
      const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
      p0 = p1;
      p1 = p2;
    }
    dp = n * (z * p1 - p0) / (z * z - 1.0);
    x[n - 1 - i] = z;  // ascending
    w[n - 1 - i] = 2.0 / ((1.0 - z * z) * dp * dp);
  }
}

}  // namespace dl
}  // namespace ntg

using namespace ntg;

extern "C" {

int ntg_dealias_create(ntg_dealias** out, ntg_plan* p, int lxd) {
  clear_error();
  NTG_CHECK_ARG(out && p, "ntg_dealias_create: null argument");
  NTG_TRY(need_metrics(p));
  if (lxd <= 0) lxd = 3 * p->lx / 2;
  NTG_TRY(dl::dispatch(p->lx, lxd, [](auto, auto) { return NTG_OK; }));
  ntg_dealias* d = new ntg_dealias();
  d->p = p;
  d->lx = p->lx;
  d->lxd = lxd;
  d->ngl = p->nelv * (int64_t)lxd * lxd * lxd;
  const int lx = p->lx;
  double xi[NTG_LXMAX], wq[NTG_LXMAX], Dm[NTG_LXMAX * NTG_LXMAX];
  gll_basis(lx, xi, wq, Dm);
  double xg[16];
  dl::gauss_legendre(lxd, xg, d->wg);
  for (int A = 0; A < lxd; ++A)
    for (int a = 0; a < lx; ++a) {
      double v = 1.0;
      for (int k = 0; k < lx; ++k)
        if (k != a) v *= (xg[A] - xi[k]) / (xi[a] - xi[k]);
      d->J[A * lx + a] = v;
    }
  // GL differentiation matrix from barycentric weights
  double lam[16];
  for (int j = 0; j < lxd; ++j) {
    double pr = 1.0;
    for (int k = 0; k < lxd; ++k)
      if (k != j) pr *= xg[j] - xg[k];
    lam[j] = 1.0 / pr;
  }
  for (int i = 0; i < lxd; ++i) {
    double diag = 0.0;
    for (int j = 0; j < lxd; ++j) {
      if (j == i) continue;
      const double v = lam[j] / lam[i] / (xg[i] - xg[j]);
      d->Dg[i * lxd + j] = v;
      diag -= v;
    }
    d->Dg[i * lxd + i] = diag;
  }
  int st = dev_alloc(&d->met_gl, (size_t)(9 * d->ngl));
  if (!st) {
    st = dl::dispatch(lx, lxd, [&](auto L, auto LD) -> int {
      constexpr int LX = decltype(L)::value, LXD = decltype(LD)::value;
      using S = dl::Smem<LX, LXD>;
      d->smem = S::BYTES;
      d->mats = std::make_shared<dl::AdvMats<LX, LXD>>(dl::adv_mats<LX, LXD>(d));
      NTG_CUDA_TRY(cudaFuncSetAttribute(dl::k_map<LX, LXD, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)S::BYTES));
      NTG_CUDA_TRY(cudaFuncSetAttribute(dl::k_map<LX, LXD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)S::BYTES));
      int occ = 0;
      NTG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, dl::k_map<LX, LXD, 0>, dl::NT, S::BYTES));
      if (occ < 1) occ = 1;
      const int64_t g = (int64_t)num_sms() * occ;
      d->grid = (int)(p->nelv < g ? p->nelv : g);
      dl::k_map<LX, LXD, 0><<<d->grid, dl::NT, S::BYTES, p->stream>>>(d->met_gl, p->met, 9, p->nelv, p->n, d->ngl,
                                                                       dl::glmat<LX, LXD>(d));
      NTG_COUNT_LAUNCH();
      NTG_CUDA_TRY(cudaGetLastError());
      return NTG_OK;
    });
  }
  if (st) {
    dev_free(d->met_gl);
    delete d;
    return st;
  }
  *out = d;
  return NTG_OK;
}

int ntg_dealias_destroy(ntg_dealias* d) {
  if (!d) return NTG_OK;
  if (d->p) cudaStreamSynchronize(d->p->stream);
  dev_free(d->met_gl);
  delete d;
  return NTG_OK;
}

int ntg_dealias_info(const ntg_dealias* d, int* lxd, int64_t* ngl) {
  clear_error();
  NTG_CHECK_ARG(d, "ntg_dealias_info: null handle");
  if (lxd) *lxd = d->lxd;
  if (ngl) *ngl = d->ngl;
  return NTG_OK;
}

int ntg_dealias_map(ntg_dealias* d, double* out_d, const double* in_d, int to_gl) {
  clear_error();
  NTG_CHECK_ARG(d && out_d && in_d, "ntg_dealias_map: null argument");
  ntg_plan* p = d->p;
  return dl::dispatch(d->lx, d->lxd, [&](auto L, auto LD) -> int {
    constexpr int LX = decltype(L)::value, LXD = decltype(LD)::value;
    if (to_gl)
      dl::k_map<LX, LXD, 0><<<d->grid, dl::NT, d->smem, p->stream>>>(out_d, in_d, 1, p->nelv, p->n, d->ngl,
                                                                      dl::glmat<LX, LXD>(d));
    else
      dl::k_map<LX, LXD, 1><<<d->grid, dl::NT, d->smem, p->stream>>>(out_d, in_d, 1, p->nelv, d->ngl, p->n,
                                                                      dl::glmat<LX, LXD>(d));
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

static int adv_dealias(ntg_dealias* d, int mode, double* f0, double* f1, double* f2, const double* vx,
                       const double* vy, const double* vz, const double* vxb, const double* vyb, const double* vzb) {
  clear_error();
  NTG_CHECK_ARG(d && f0 && f1 && f2 && vx && vy && vz && vxb && vyb && vzb, "dealiased advection: null argument");
  ntg_plan* p = d->p;
  return dl::dispatch(d->lx, d->lxd, [&](auto L, auto LD) -> int {
    constexpr int LX = decltype(L)::value, LXD = decltype(LD)::value;
    using S = dl::AdvShape<LX, LXD>;
    const auto& P = *static_cast<const dl::AdvMats<LX, LXD>*>(d->mats.get());
    const int64_t g = (p->nelv + S::EPB - 1) / S::EPB, cap = (int64_t)num_sms() * S::MINB;
    const int grid = (int)(g < cap ? g : cap);
    if (mode == 0) {
      NTG_TRY((fx::use_smem<dl::k_adv<LX, LXD, 0>>(S::SMEM)));
      dl::k_adv<LX, LXD, 0><<<grid, S::NT, S::SMEM, p->stream>>>(f0, f1, f2, vx, vy, vz, vxb, vyb, vzb, d->met_gl,
                                                                 d->ngl, p->nelv, P);
    } else {
      NTG_TRY((fx::use_smem<dl::k_adv<LX, LXD, 1>>(S::SMEM)));
      dl::k_adv<LX, LXD, 1><<<grid, S::NT, S::SMEM, p->stream>>>(f0, f1, f2, vx, vy, vz, vxb, vyb, vzb, d->met_gl,
                                                                 d->ngl, p->nelv, P);
    }
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

int ntg_adjoint_advection_dealias(ntg_dealias* d, double* fx_d, double* fy_d, double* fz_d, const double* vx_d,
                                  const double* vy_d, const double* vz_d, const double* vxb_d, const double* vyb_d,
                                  const double* vzb_d) {
  return adv_dealias(d, 0, fx_d, fy_d, fz_d, vx_d, vy_d, vz_d, vxb_d, vyb_d, vzb_d);
}

int ntg_linear_advection_dealias(ntg_dealias* d, double* fx_d, double* fy_d, double* fz_d, const double* vx_d,
                                 const double* vy_d, const double* vz_d, const double* vxb_d, const double* vyb_d,
                                 const double* vzb_d) {
  return adv_dealias(d, 1, fx_d, fy_d, fz_d, vx_d, vy_d, vz_d, vxb_d, vyb_d, vzb_d);
}

}  // extern "C"
