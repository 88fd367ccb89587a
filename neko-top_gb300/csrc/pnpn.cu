// Pn/Pn splitting residuals on either side of the pressure and velocity
// solves (FP64), as the adjoint/forward step calls them
// (sources/adjoint/adjoint_pnpn.f90:716-723 prs_res%compute and :747-753
// vel_res%compute):
//
//   pressure  wa = curl(curl(u_e)),  ta_d = Binv gs(f_d / rho - (mu / rho) B wa_d)
//             p_res = -A(h1 = 1/rho) p + sum_d cdtp_d(ta_d)
//                     - (bd/dt) sum_c u_c s_c   on velocity-surface nodes
//                     - sum_c ta_c s'_c         on symmetry-surface nodes
//   velocity  u_res_c = f_c - (mu K + rho (bd/dt) B) u_c - opgrad_c(p)
//
// (s, s': outward normal times facet area, per surface node, from the
// caller.)  Neither residual is gs-assembled or masked: the caller does that
// next, as the reference does.
//
// Fusion: the pressure residual's Laplacian of p and its three cdtp terms
// are one element-tile pass (both end in the transposed reference
// derivatives, so their r/s/t fluxes are summed before one D^T contraction);
// the velocity residual computes all three components and the pressure
// gradient in one pass, so G, B and the cofactors are read once instead of
// three times.  The contractions run in fixed point (fx.cuh) and the
// gather-scatters take three fields a launch: both residuals of 24^3 elements,
// lx = 8, take 2.5 ms where FP64 sums took 7.1.  mu and rho are fields or constants (null pointer -> the
// constant).
#include "deriv.cuh"

namespace ntg {
namespace pn {

using dv::DMat;
using dv::FxShape;

struct GPtr {
  const double* g[6];
};

// mu and rho: fields, or constants (ri: the constant's reciprocal)
struct Coefs {
  const double* mu;
  const double* rho;
  double muc, rhoc, ri;
};

// X_c holds gs(B curl t)_c; becomes f_c / rho - (mu / rho) B (Binv X_c)
__global__ void k_ta(double* __restrict__ x0, double* __restrict__ x1, double* __restrict__ x2,
                     const double* __restrict__ f0, const double* __restrict__ f1, const double* __restrict__ f2,
                     const double* __restrict__ B, const double* __restrict__ binv, Coefs c, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const double ri = c.rho ? 1.0 / c.rho[q] : c.ri;
    const double m = (c.mu ? c.mu[q] : c.muc) * ri * (B[q] * binv[q]);
    x0[q] = fma(-m, x0[q], f0[q] * ri);
    x1[q] = fma(-m, x1[q], f1[q] * ri);
    x2[q] = fma(-m, x2[q], f2[q] * ri);
  }
}

// p_res = -D^T (h1 G D p) + sum_d cdtp_d(binv ta_d), h1 = 1 / rho
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 4>::NT, FxShape<LX, 4>::MINB)
    k_prs_core(double* __restrict__ pres, const double* __restrict__ pp, const double* __restrict__ ta0,
               const double* __restrict__ ta1, const double* __restrict__ ta2, const double* __restrict__ binv,
               Coefs c, int64_t nelv, const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
               GPtr G, const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(4)
  dv::stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    NTG_FX_NODES { NTG_FX_NODE T[p] = pp[q]; }
    __syncthreads();
    NTG_FX_LINES { NTG_FX_LINE fx::deriv_line<LX>(P.D, P.d, T, T + (1 + d) * TS, d, lq, false); }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      const double ur = T[TS + p], us = T[2 * TS + p], ut = T[3 * TS + p];
      const double h1 = c.rho ? 1.0 / c.rho[q] : c.ri, b = w3t[node] * binv[q];
      const double a0 = b * ta0[q], a1 = b * ta1[q], a2 = b * ta2[q];
      const double g12 = G.g[1][q], g13 = G.g[2][q], g23 = G.g[4][q];
      const double er = G.g[0][q] * ur + g12 * us + g13 * ut, es = g12 * ur + G.g[3][q] * us + g23 * ut;
      const double et = g13 * ur + g23 * us + G.g[5][q] * ut;
      T[TS + p] = fma(-h1, er, met[0 * n + q] * a0 + met[1 * n + q] * a1 + met[2 * n + q] * a2);
      T[2 * TS + p] = fma(-h1, es, met[3 * n + q] * a0 + met[4 * n + q] * a1 + met[5 * n + q] * a2);
      T[3 * TS + p] = fma(-h1, et, met[6 * n + q] * a0 + met[7 * n + q] * a1 + met[8 * n + q] * a2);
    }
    __syncthreads();
    NTG_FX_LINES {
      NTG_FX_LINE
      fx::flux_line<LX>(P.DT, P.dt, T + (1 + d) * TS, reinterpret_cast<int*>(T + 4 * TS) + r, d, lq);
    }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      pres[q] = fx::flux_sum<LX>(T + TS, T + 2 * TS, T + 3 * TS, reinterpret_cast<const int*>(T + 4 * TS), node);
    }
  }
}

// res_c = f_c - D^T (mu G D u_c) - rho (bd/dt) B u_c - opgrad_c(p), c = 0..2.
// P.DT carries mus, a constant mu (1 when mu is a field, which then
// multiplies the fluxes).
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 7>::NT, FxShape<LX, 7>::MINB)
    k_vel_res(double* __restrict__ r0, double* __restrict__ r1, double* __restrict__ r2,
              const double* __restrict__ u0, const double* __restrict__ u1, const double* __restrict__ u2,
              const double* __restrict__ pp, const double* __restrict__ f0, const double* __restrict__ f1,
              const double* __restrict__ f2, Coefs c, double mus, double bddt, int64_t nelv,
              const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P, GPtr G,
              const double* __restrict__ B, const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(7)
  dv::stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    // tiles 0-2: the gradient of p; 3: a component; 4-6: its derivatives, then fluxes
    NTG_FX_NODES { NTG_FX_NODE T[3 * TS + p] = pp[q]; }
    __syncthreads();
    NTG_FX_LINES { NTG_FX_LINE fx::deriv_line<LX>(P.D, P.d, T + 3 * TS, T + d * TS, d, lq); }
#pragma unroll 1
    for (int cc = 0; cc < 3; ++cc) {
      const double* u = cc == 0 ? u0 : cc == 1 ? u1 : u2;
      const double* f = cc == 0 ? f0 : cc == 1 ? f1 : f2;
      double* res = cc == 0 ? r0 : cc == 1 ? r1 : r2;
      __syncthreads();
      NTG_FX_NODES { NTG_FX_NODE T[3 * TS + p] = u[q]; }
      __syncthreads();
      NTG_FX_LINES { NTG_FX_LINE fx::deriv_line<LX>(P.D, P.d, T + 3 * TS, T + (4 + d) * TS, d, lq, false); }
      __syncthreads();
      NTG_FX_NODES {
        NTG_FX_NODE
        const double ur = T[4 * TS + p], us = T[5 * TS + p], ut = T[6 * TS + p];
        const double g12 = G.g[1][q], g13 = G.g[2][q], g23 = G.g[4][q];
        T[4 * TS + p] = G.g[0][q] * ur + g12 * us + g13 * ut;
        T[5 * TS + p] = g12 * ur + G.g[3][q] * us + g23 * ut;
        T[6 * TS + p] = g13 * ur + g23 * us + G.g[5][q] * ut;
      }
      if (c.mu || mus != 1.0) {  // a field, or a constant too large or small for P.DT
        NTG_FX_NODES {
          NTG_FX_NODE
          const double m = c.mu ? c.mu[q] : mus;
          T[4 * TS + p] *= m;
          T[5 * TS + p] *= m;
          T[6 * TS + p] *= m;
        }
      }
      __syncthreads();
      NTG_FX_LINES {
        NTG_FX_LINE
        fx::flux_line<LX>(P.DT, P.dt, T + (4 + d) * TS, reinterpret_cast<int*>(T + 7 * TS) + r, d, lq, c.mu != nullptr);
      }
      __syncthreads();
      NTG_FX_NODES {
        NTG_FX_NODE
        const double h2 = (c.rho ? c.rho[q] : c.rhoc) * bddt;
        const double gp = met[cc * n + q] * T[p] + met[(3 + cc) * n + q] * T[TS + p] + met[(6 + cc) * n + q] * T[2 * TS + p];
        const double s = fx::flux_sum<LX>(T + 4 * TS, T + 5 * TS, T + 6 * TS,
                                          reinterpret_cast<const int*>(T + 7 * TS), node);
        res[q] = fma(-w3t[node], gp, f[q]) - fma(h2 * B[q], T[3 * TS + p], s);
      }
    }
    __syncthreads();
  }
}

// res[q] -= scale sum_c (mul[q]) v_c[q] s_c[t] over the surface entries t
__global__ void k_surface(double* __restrict__ res, const int32_t* __restrict__ idx, const double* __restrict__ s,
                          int64_t ns, int base, const double* __restrict__ v0, const double* __restrict__ v1,
                          const double* __restrict__ v2, const double* __restrict__ mul, double scale, int64_t n) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ns; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = (int64_t)idx[t] - base;
    if (q < 0 || q >= n) continue;
    const double m = mul ? mul[q] : 1.0;
    res[q] -= scale * (m * v0[q] * s[t] + m * v1[q] * s[ns + t] + m * v2[q] * s[2 * ns + t]);
  }
}

GPtr gptr(const ntg_plan* p) {
  GPtr G;
  for (int a = 0; a < 6; ++a) G.g[a] = p->g[a];
  return G;
}

}  // namespace pn
}  // namespace ntg

using namespace ntg;

extern "C" {

int ntg_pnpn_prs_res(ntg_plan* p, double* p_res, const double* pr, const double* u, const double* v, const double* w,
                     const double* ue, const double* ve, const double* we, const double* fx, const double* fy,
                     const double* fz, const double* mu_d, double mu_c, const double* rho_d, double rho_c, double bd,
                     double dt, const int32_t* prs_idx, const double* prs_s, int64_t nprs, const int32_t* sym_idx,
                     const double* sym_s, int64_t nsym, int base) {
  clear_error();
  NTG_CHECK_ARG(p && p_res && pr && u && v && w && ue && ve && we && fx && fy && fz,
                "ntg_pnpn_prs_res: null field argument");
  NTG_CHECK_ARG(nprs >= 0 && nsym >= 0 && (nprs == 0 || (prs_idx && prs_s)) && (nsym == 0 || (sym_idx && sym_s)),
                "ntg_pnpn_prs_res: bad surface list");
  NTG_CHECK_ARG(dt > 0.0 && (rho_d || rho_c != 0.0), "ntg_pnpn_prs_res: need dt > 0 and rho != 0");
  NTG_TRY(need_metrics(p));
  const int64_t n = p->n;
  double* t = plan_scratch(p, 6 * n);
  if (!t) return NTG_ERR_ALLOC;
  double *t0 = t, *t1 = t + n, *t2 = t + 2 * n, *x0 = t + 3 * n, *x1 = t + 4 * n, *x2 = t + 5 * n;
  cudaStream_t s = p->stream;
  const pn::Coefs c{mu_d, rho_d, mu_c, rho_c, rho_d ? 1.0 : 1.0 / rho_c};
  // Binv t = curl(u_e), its Binv applied where t is read; X = gs(B curl(Binv t))
  NTG_TRY(curl_gs(p, t0, t1, t2, ue, ve, we, nullptr));
  NTG_TRY(curl_gs(p, x0, x1, x2, t0, t1, t2, p->binv));
  // ta = gs(f / rho - (mu / rho) B wa); its Binv is applied where ta is read
  { pn::k_ta<<<grid_for(n, 256), 256, 0, s>>>(x0, x1, x2, fx, fy, fz, p->B, p->binv, c, n); NTG_COUNT_LAUNCH(); }
  NTG_TRY(gs_launch3(p, x0, x1, x2, s));
  NTG_TRY(dv::dispatch<4>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 4>;
    NTG_TRY(fx::use_smem<pn::k_prs_core<LX>>(S::SMEM));
    pn::k_prs_core<LX><<<dv::fx_grid<LX, 4>(p), S::NT, S::SMEM, s>>>(
        p_res, pr, x0, x1, x2, p->binv, c, p->nelv, dv::dmat<LX>(p), fx::plan_mats<LX>(p, 1.0), pn::gptr(p), p->met,
        n);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  }));
  if (nprs) {
    pn::k_surface<<<grid_for(nprs, 256), 256, 0, s>>>(p_res, prs_idx, prs_s, nprs, base, u, v, w, nullptr, bd / dt,
                                                      n);
    NTG_COUNT_LAUNCH();
  }
  if (nsym) {
    pn::k_surface<<<grid_for(nsym, 256), 256, 0, s>>>(p_res, sym_idx, sym_s, nsym, base, x0, x1, x2, p->binv, 1.0,
                                                      n);
    NTG_COUNT_LAUNCH();
  }
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

int ntg_pnpn_vel_res(ntg_plan* p, double* u_res, double* v_res, double* w_res, const double* u, const double* v,
                     const double* w, const double* pr, const double* fx, const double* fy, const double* fz,
                     const double* mu_d, double mu_c, const double* rho_d, double rho_c, double bd, double dt) {
  clear_error();
  NTG_CHECK_ARG(p && u_res && v_res && w_res && u && v && w && pr && fx && fy && fz,
                "ntg_pnpn_vel_res: null field argument");
  NTG_CHECK_ARG(dt > 0.0, "ntg_pnpn_vel_res: need dt > 0");
  NTG_TRY(need_metrics(p));
  const pn::Coefs c{mu_d, rho_d, mu_c, rho_c, 0.0};
  const double fold = !mu_d && fx::foldable(mu_c) ? mu_c : 1.0;  // a constant mu goes into D^T
  const double mus = mu_d || fold == mu_c ? 1.0 : mu_c;
  return dv::dispatch<7>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 7>;
    NTG_TRY(fx::use_smem<pn::k_vel_res<LX>>(S::SMEM));
    pn::k_vel_res<LX><<<dv::fx_grid<LX, 7>(p), S::NT, S::SMEM, p->stream>>>(
        u_res, v_res, w_res, u, v, w, pr, fx, fy, fz, c, mus, bd / dt, p->nelv, dv::dmat<LX>(p),
        fx::plan_mats<LX>(p, fold), pn::gptr(p), p->B, p->met, p->n);
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

}  // extern "C"
