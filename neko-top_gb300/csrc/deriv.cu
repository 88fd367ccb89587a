// Spectral-element derivative operators (FP64) and the adjoint-equation
// terms built on them:
//
//   metrics      drdx .. dtdz (cofactors of dx/dr) and 1/jac from the coordinates
//   dudxyz       strong derivative (dr u_r + ds u_s + dt u_t) / jac   (Neko dudxyz)
//   opgrad       weak gradient w3 (drdx u_r + dsdx u_s + dtdx u_t), ... (= B grad u)
//   cdtp         D_r^T (w3 dr x) + D_s^T (w3 ds x) + D_t^T (w3 dt x) (transpose of opgrad)
//   conv1        vx du/dx + vy du/dy + vz du/dz (strong, pointwise)
//   curl         strong curl averaged across element copies: Binv gs(B curl u)
//
//   adjoint advection (no dealiasing), sources/adjoint/adv_adjoint_no_dealias.f90:118-302:
//       f_i -= sum_j u_j opgrad_i(Ub_j) + sum_d cdtp_d(u_i Ub_d)
//     (the device branch there; its CPU branch adds two of the three cdtp terms)
//   linearised advection (no dealiasing), same file :331-400:
//       f_i -= B conv1(u_i; Ub) + B conv1(Ub_i; u)
//   minimum-dissipation adjoint forcing,
//   sources/source_terms/adjoint_minimum_dissipation_source_term.f90:175-249:
//       f += scale curl(curl(u)), kept inside a zone (mask_exterior_const,
//       sources/neko_ext/mask_ops.f90:55-82) when one is given
//
// Layout: element tiles in shared memory; contractions in fixed point
// (fx.cuh), everything else FP64 (these feed the adjoint right-hand sides
// and sensitivities).
#include "deriv.cuh"

namespace ntg {
namespace dv {

// 9 cofactors (drdx, drdy, drdz, dsdx, ..., dtdz) and 1/jac, stored m * n + l
template <int LX>
__global__ void __launch_bounds__(Shape<LX, 3>::THREADS)
    k_metrics(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z, int64_t nelv,
              const __grid_constant__ DMat<LX> M, double* __restrict__ met, int64_t n) {
  using S = Shape<LX, 3>;
  constexpr int LX2 = S::LX2, LX3 = S::LX3, EPB = S::EPB;
  __shared__ double sx[EPB][LX3], sy[EPB][LX3], sz[EPB][LX3];
  const int tid = threadIdx.x, le = tid / LX2, ij = tid - le * LX2, i = ij % LX, j = ij / LX;
  const bool worker = tid < S::NW;
  for (int64_t g = blockIdx.x; g * EPB < nelv; g += gridDim.x) {
    const int64_t e = g * EPB + le;
    const bool act = worker && e < nelv;
    for (int k = 0; k < LX && worker; ++k) {
      const int64_t q = e * LX3 + k * LX2 + ij;
      sx[le][k * LX2 + ij] = act ? x[q] : 0.0;
      sy[le][k * LX2 + ij] = act ? y[q] : 0.0;
      sz[le][k * LX2 + ij] = act ? z[q] : 0.0;
    }
    __syncthreads();
    if (act) {
      for (int k = 0; k < LX; ++k) {
        double xr, xs, xt, yr, ys, yt, zr, zs, zt;
        rgrad<LX>(sx[le], M, i, j, k, xr, xs, xt);
        rgrad<LX>(sy[le], M, i, j, k, yr, ys, yt);
        rgrad<LX>(sz[le], M, i, j, k, zr, zs, zt);
        const double c[9] = {ys * zt - yt * zs, xt * zs - xs * zt, xs * yt - xt * ys,
                             yt * zr - yr * zt, xr * zt - xt * zr, xt * yr - xr * yt,
                             yr * zs - ys * zr, xs * zr - xr * zs, xr * ys - xs * yr};
        const double jac = xr * c[0] + yr * c[1] + zr * c[2];
        const int64_t q = e * LX3 + k * LX2 + ij;
#pragma unroll
        for (int m = 0; m < 9; ++m) met[m * n + q] = c[m];
        met[9 * n + q] = 1.0 / jac;
      }
    }
    __syncthreads();
  }
}

// Gradient of u with the cofactors: out_d = (strong) or w3 * (weak)
// derivative, for the non-null out_d.
template <int LX, bool WEAK>
__global__ void __launch_bounds__(FxShape<LX, 4>::NT, FxShape<LX, 4>::MINB)
    k_grad(double* __restrict__ o0, double* __restrict__ o1, double* __restrict__ o2, const double* __restrict__ u,
           int64_t nelv, const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
           const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(4)
  if (WEAK) stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    NTG_FX_NODES { NTG_FX_NODE T[p] = u[q]; }
    __syncthreads();
    NTG_FX_LINES { NTG_FX_LINE fx::deriv_line<LX>(P.D, P.d, T, T + (1 + d) * TS, d, lq); }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      const double ur = T[TS + p], us = T[2 * TS + p], ut = T[3 * TS + p];
      const double sc = WEAK ? w3t[node] : met[9 * n + q];
      if (o0) o0[q] = sc * (met[q] * ur + met[3 * n + q] * us + met[6 * n + q] * ut);
      if (o1) o1[q] = sc * (met[n + q] * ur + met[4 * n + q] * us + met[7 * n + q] * ut);
      if (o2) o2[q] = sc * (met[2 * n + q] * ur + met[5 * n + q] * us + met[8 * n + q] * ut);
    }
  }
}

// out = cdtp of x with the cofactors of direction dir
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 3>::NT, FxShape<LX, 3>::MINB)
    k_cdtp(double* __restrict__ out, const double* __restrict__ x, int dir, int64_t nelv,
           const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
           const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(3)
  stage_w3<LX>(w3t, M, NT);
  __syncthreads();
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    NTG_FX_NODES {
      NTG_FX_NODE
      const double a = w3t[node] * x[q];
      T[p] = met[dir * n + q] * a;
      T[TS + p] = met[(3 + dir) * n + q] * a;
      T[2 * TS + p] = met[(6 + dir) * n + q] * a;
    }
    __syncthreads();
    NTG_FX_LINES {
      NTG_FX_LINE
      fx::flux_line<LX>(P.DT, P.dt, T + d * TS, reinterpret_cast<int*>(T + 3 * TS) + r, d, lq);
    }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      out[q] = fx::flux_sum<LX>(T, T + TS, T + 2 * TS, reinterpret_cast<const int*>(T + 3 * TS), node);
    }
    __syncthreads();
  }
}

// out = v . grad(a) (conv1, strong)
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 4>::NT, FxShape<LX, 4>::MINB)
    k_conv(double* __restrict__ out, const double* __restrict__ a, const double* __restrict__ v0,
           const double* __restrict__ v1, const double* __restrict__ v2, int64_t nelv,
           const __grid_constant__ fx::Mats<LX> P, const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(4)
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    NTG_FX_NODES { NTG_FX_NODE T[p] = a[q]; }
    __syncthreads();
    NTG_FX_LINES { NTG_FX_LINE fx::deriv_line<LX>(P.D, P.d, T, T + (1 + d) * TS, d, lq); }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      const double x = v0[q], y = v1[q], z = v2[q];
      double acc = 0.0;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        acc = fma(met[3 * d * n + q] * x + met[(3 * d + 1) * n + q] * y + met[(3 * d + 2) * n + q] * z,
                  T[(1 + d) * TS + p], acc);
      out[q] = acc * met[9 * n + q];
    }
  }
}

// B curl(u) (strong curl times B = w3 * cofactor combinations); scale: null,
// or a factor per node that multiplies u first
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 9>::NT, FxShape<LX, 9>::MINB)
    k_curl(double* __restrict__ w0, double* __restrict__ w1, double* __restrict__ w2, const double* __restrict__ ux,
           const double* __restrict__ uy, const double* __restrict__ uz, const double* __restrict__ scale,
           int64_t nelv, const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
           const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(9)
  stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    if (scale) {
      NTG_FX_NODES {
        NTG_FX_NODE
        const double b = scale[q];
        T[p] = ux[q] * b;
        T[TS + p] = uy[q] * b;
        T[2 * TS + p] = uz[q] * b;
      }
    } else {
      NTG_FX_NODES {
        NTG_FX_NODE
        T[p] = ux[q];
        T[TS + p] = uy[q];
        T[2 * TS + p] = uz[q];
      }
    }
#pragma unroll 1
    for (int dir = 0; dir < 3; ++dir) {
      __syncthreads();
      NTG_FX_LINES {
        NTG_FX_LINE  // d: the field here
        fx::deriv_line<LX>(P.D, P.d, T + d * TS, T + (3 + d) * TS, dir, lq);
      }
      __syncthreads();
      NTG_FX_NODES {
        NTG_FX_NODE
        const double gx = T[3 * TS + p], gy = T[4 * TS + p], gz = T[5 * TS + p];
        const double c0 = met[3 * dir * n + q], c1 = met[(3 * dir + 1) * n + q], c2 = met[(3 * dir + 2) * n + q];
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
        if (dir > 0) {
          a0 = T[6 * TS + p];
          a1 = T[7 * TS + p];
          a2 = T[8 * TS + p];
        }
        a0 = fma(c1, gz, fma(-c2, gy, a0));
        a1 = fma(c2, gx, fma(-c0, gz, a1));
        a2 = fma(c0, gy, fma(-c1, gx, a2));
        if (dir < 2) {
          T[6 * TS + p] = a0;
          T[7 * TS + p] = a1;
          T[8 * TS + p] = a2;
        } else {
          const double w3 = w3t[node];
          w0[q] = w3 * a0;
          w1[q] = w3 * a1;
          w2[q] = w3 * a2;
        }
      }
    }
    __syncthreads();
  }
}

// The adjoint advection without dealiasing in one element pass:
//   f_i -= sum_j u_j opgrad_i(Ub_j) + sum_d cdtp_d(u_i Ub_d).
// With a_d = sum_j u_j dUb_j/dr_d the first sum is w3 sum_d c_di a_d (18
// products per node where mixing each gradient first takes 36); the second
// shares the contravariant velocity V_d = sum_c c_dc Ub_c between the three
// components, and the weights come out of D^T: D_d^T (w3 f) = w3 (DT_d f)
// with DT = W^-1 D^T W.  42 FP64 operations per node (198 with the
// contractions on the FP64 pipe).
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 9>::NT, FxShape<LX, 9>::MINB)
    k_adv_adj_nd(double* __restrict__ f0, double* __restrict__ f1, double* __restrict__ f2,
                 const double* __restrict__ u0, const double* __restrict__ u1, const double* __restrict__ u2,
                 const double* __restrict__ b0, const double* __restrict__ b1, const double* __restrict__ b2,
                 int64_t nelv, const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
                 const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(9)
  stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    // tiles 0-2: Ub, then V; 3-5: u, then fluxes; 6-8: a_d, then the opgrad part
    NTG_FX_NODES {
      NTG_FX_NODE
      T[p] = b0[q];
      T[TS + p] = b1[q];
      T[2 * TS + p] = b2[q];
      T[3 * TS + p] = u0[q];
      T[4 * TS + p] = u1[q];
      T[5 * TS + p] = u2[q];
    }
    __syncthreads();
    // a_d along its lines: the three fields' derivatives of one line each are
    // weighted by u and summed in registers
    NTG_FX_LINES {
      NTG_FX_LINE
      const int b = TL::base(d, lq), st = TL::stride(d);
      double a[LX];
#pragma unroll
      for (int l = 0; l < LX; ++l) a[l] = 0.0;
#pragma unroll 1
      for (int f = 0; f < 3; ++f) {
        const double *v = T + f * TS + b, *u = T + (3 + f) * TS + b;
        double x[LX];
#pragma unroll
        for (int l = 0; l < LX; ++l) x[l] = v[l * st];
        fx::line_dbl<LX, LX, true>(P.D, P.d, x, true, [&](int A, double y) { a[A] = fma(y, u[A * st], a[A]); });
      }
#pragma unroll
      for (int l = 0; l < LX; ++l) T[(6 + d) * TS + b + l * st] = a[l];
    }
    __syncthreads();
    NTG_FX_NODES {
      NTG_FX_NODE
      double m[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) m[c] = met[c * n + q];
      const double bx = T[p], by = T[TS + p], bz = T[2 * TS + p];
      const double ar = T[6 * TS + p], as = T[7 * TS + p], at = T[8 * TS + p];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T[c * TS + p] = m[3 * c] * bx + m[3 * c + 1] * by + m[3 * c + 2] * bz;
        T[(6 + c) * TS + p] = m[c] * ar + m[3 + c] * as + m[6 + c] * at;
      }
    }
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      const double* uc = c == 0 ? u0 : c == 1 ? u1 : u2;
      double* fc = c == 0 ? f0 : c == 1 ? f1 : f2;
      NTG_FX_NODES {
        NTG_FX_NODE
        const double v = uc[q];
        T[3 * TS + p] = v * T[p];
        T[4 * TS + p] = v * T[TS + p];
        T[5 * TS + p] = v * T[2 * TS + p];
      }
      __syncthreads();
      NTG_FX_LINES {
        NTG_FX_LINE
        fx::flux_line<LX>(P.DT, P.dt, T + (3 + d) * TS, reinterpret_cast<int*>(T + 9 * TS) + r, d, lq);
      }
      __syncthreads();
      NTG_FX_NODES {
        NTG_FX_NODE
        const double s = fx::flux_sum<LX>(T + 3 * TS, T + 4 * TS, T + 5 * TS,
                                          reinterpret_cast<const int*>(T + 9 * TS), node);
        fc[q] = fma(-w3t[node], s + T[(6 + c) * TS + p], fc[q]);
      }
    }
    __syncthreads();
  }
}

// The linearised advection without dealiasing in one element pass:
//   f_i -= B conv1(u_i; Ub) + B conv1(Ub_i; u)
//        = w3 sum_d (V_d(Ub) du_i/dr_d + V_d(u) dUb_i/dr_d),
// V_d(x) = sum_c c_dc x_c: 39 FP64 operations per node (216 with the
// contractions on the FP64 pipe).
template <int LX>
__global__ void __launch_bounds__(FxShape<LX, 9>::NT, FxShape<LX, 9>::MINB)
    k_adv_lin_nd(double* __restrict__ f0, double* __restrict__ f1, double* __restrict__ f2,
                 const double* __restrict__ u0, const double* __restrict__ u1, const double* __restrict__ u2,
                 const double* __restrict__ b0, const double* __restrict__ b1, const double* __restrict__ b2,
                 int64_t nelv, const __grid_constant__ DMat<LX> M, const __grid_constant__ fx::Mats<LX> P,
                 const double* __restrict__ met, int64_t n) {
  NTG_FX_PROLOGUE(9)
  stage_w3<LX>(w3t, M, NT);
  NTG_FX_ELEMENTS {
    NTG_FX_NE;
    // tiles 0-2: the velocity differentiated; 3-5: V_d of the other; 6-8: sums
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      const double *x0 = pass ? b0 : u0, *x1 = pass ? b1 : u1, *x2 = pass ? b2 : u2;
      const double *y0 = pass ? u0 : b0, *y1 = pass ? u1 : b1, *y2 = pass ? u2 : b2;
      NTG_FX_NODES {
        NTG_FX_NODE
        const double x = x0[q], y = x1[q], z = x2[q];
        T[p] = y0[q];
        T[TS + p] = y1[q];
        T[2 * TS + p] = y2[q];
        if (pass == 0) T[6 * TS + p] = T[7 * TS + p] = T[8 * TS + p] = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c)
          T[(3 + c) * TS + p] = met[3 * c * n + q] * x + met[(3 * c + 1) * n + q] * y + met[(3 * c + 2) * n + q] * z;
      }
      __syncthreads();
#pragma unroll 1
      for (int dir = 0; dir < 3; ++dir) {
        NTG_FX_LINES {
          NTG_FX_LINE  // d: the field here
          const int b = TL::base(dir, lq), st = TL::stride(dir);
          const double *in = T + d * TS + b, *v = T + (3 + dir) * TS + b;
          double* o = T + (6 + d) * TS + b;
          double x[LX];
#pragma unroll
          for (int l = 0; l < LX; ++l) x[l] = in[l * st];
          fx::line_dbl<LX, LX, true>(P.D, P.d, x, true, [&](int A, double y) {
            o[A * st] = fma(y, v[A * st], o[A * st]);
          });
        }
        __syncthreads();
      }
    }
    NTG_FX_NODES {
      NTG_FX_NODE
      const double w = -w3t[node];
      f0[q] = fma(w, T[6 * TS + p], f0[q]);
      f1[q] = fma(w, T[7 * TS + p], f1[q]);
      f2[q] = fma(w, T[8 * TS + p], f2[q]);
    }
    // the next element's first nodes write tiles 0-5, read last before the
    // barrier above, and each thread's own nodes of tiles 6-8
  }
}

// a, b, c *= s
__global__ void k_mul3(double* __restrict__ a, double* __restrict__ b, double* __restrict__ c,
                       const double* __restrict__ s, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const double f = s[q];
    a[q] *= f;
    b[q] *= f;
    c[q] *= f;
  }
}

__global__ void k_inv(double* __restrict__ a, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    a[q] = 1.0 / a[q];
}

// f_c += scale binv w_c on all nodes (zone null) or on the zone's nodes only
__global__ void k_add_zone(double* __restrict__ f0, double* __restrict__ f1, double* __restrict__ f2,
                           const double* __restrict__ w0, const double* __restrict__ w1,
                           const double* __restrict__ w2, const double* __restrict__ binv, double scale,
                           const int32_t* __restrict__ zone, int64_t nzone, int base, int64_t n) {
  const int64_t cnt = zone ? nzone : n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < cnt; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = zone ? (int64_t)zone[t] - base : t;
    if (q < 0 || q >= n) continue;
    const double b = binv[q];
    f0[q] = fma(scale, w0[q] * b, f0[q]);
    f1[q] = fma(scale, w1[q] * b, f1[q]);
    f2[q] = fma(scale, w2[q] * b, f2[q]);
  }
}

}  // namespace dv

double* plan_scratch(ntg_plan* p, int64_t count) {
  if (p->dscr_n < count) {
    // the stream may still use the old buffer
    if (p->dscr && cudaStreamSynchronize(p->stream) != cudaSuccess) return nullptr;
    dev_free(p->dscr);
    p->dscr_n = 0;
    if (dev_alloc(&p->dscr, (size_t)count)) return nullptr;
    p->dscr_n = count;
  }
  return p->dscr;
}

// w = gs(B curl(scale u)); scale null: 1
int curl_gs(ntg_plan* p, double* w0, double* w1, double* w2, const double* ux, const double* uy, const double* uz,
            const double* scale) {
  cudaStream_t s = p->stream;
  NTG_TRY(dv::dispatch<9>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 9>;
    NTG_TRY(fx::use_smem<dv::k_curl<LX>>(S::SMEM));
    dv::k_curl<LX><<<dv::fx_grid<LX, 9>(p), S::NT, S::SMEM, s>>>(w0, w1, w2, ux, uy, uz, scale, p->nelv,
                                                                 dv::dmat<LX>(p), fx::plan_mats<LX>(p, 1.0), p->met,
                                                                 p->n);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  }));
  NTG_TRY(gs_launch3(p, w0, w1, w2, s));
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

// w = Binv gs(B curl u)
static int curl_avg(ntg_plan* p, double* w0, double* w1, double* w2, const double* ux, const double* uy,
                    const double* uz) {
  NTG_TRY(curl_gs(p, w0, w1, w2, ux, uy, uz, nullptr));
  { dv::k_mul3<<<grid_for(p->n, 256), 256, 0, p->stream>>>(w0, w1, w2, p->binv, p->n); NTG_COUNT_LAUNCH(); }
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

}  // namespace ntg

using namespace ntg;

extern "C" {

int ntg_metrics_set(ntg_plan* p, const double* x_d, const double* y_d, const double* z_d) {
  clear_error();
  NTG_CHECK_ARG(p && x_d && y_d && z_d, "ntg_metrics_set: null argument");
  if (!p->met) NTG_TRY(dev_alloc(&p->met, (size_t)p->n * 10));
  if (!p->binv) NTG_TRY(dev_alloc(&p->binv, (size_t)p->n));
  cudaStream_t s = p->stream;
  NTG_TRY(dv::dispatch<3>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    dv::k_metrics<LX><<<dv::grid_of<LX, 3>(p), dv::Shape<LX, 3>::THREADS, 0, s>>>(x_d, y_d, z_d, p->nelv,
                                                                                    dv::dmat<LX>(p), p->met, p->n);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  }));
  NTG_CUDA_TRY(cudaMemcpyAsync(p->binv, p->B, sizeof(double) * p->n, cudaMemcpyDeviceToDevice, s));
  NTG_TRY(gs_launch(p, p->binv, NTG_GS_ADD, s));
  { dv::k_inv<<<grid_for(p->n, 256), 256, 0, s>>>(p->binv, p->n); NTG_COUNT_LAUNCH(); }
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

int ntg_dudxyz(ntg_plan* p, double* du_d, const double* u_d, int dir) {
  clear_error();
  NTG_CHECK_ARG(p && du_d && u_d && dir >= 0 && dir <= 2, "ntg_dudxyz: bad argument");
  NTG_TRY(need_metrics(p));
  double* o[3] = {nullptr, nullptr, nullptr};
  o[dir] = du_d;
  return dv::dispatch<1>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 4>;
    NTG_TRY((fx::use_smem<dv::k_grad<LX, false>>(S::SMEM)));
    dv::k_grad<LX, false><<<dv::fx_grid<LX, 4>(p), S::NT, S::SMEM, p->stream>>>(
        o[0], o[1], o[2], u_d, p->nelv, dv::dmat<LX>(p), fx::plan_mats<LX>(p, 1.0), p->met, p->n);
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

int ntg_opgrad(ntg_plan* p, double* ux_d, double* uy_d, double* uz_d, const double* u_d) {
  clear_error();
  NTG_CHECK_ARG(p && ux_d && uy_d && uz_d && u_d, "ntg_opgrad: null argument");
  NTG_TRY(need_metrics(p));
  return dv::dispatch<1>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 4>;
    NTG_TRY((fx::use_smem<dv::k_grad<LX, true>>(S::SMEM)));
    dv::k_grad<LX, true><<<dv::fx_grid<LX, 4>(p), S::NT, S::SMEM, p->stream>>>(
        ux_d, uy_d, uz_d, u_d, p->nelv, dv::dmat<LX>(p), fx::plan_mats<LX>(p, 1.0), p->met, p->n);
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

int ntg_cdtp(ntg_plan* p, double* dtx_d, const double* x_d, int dir) {
  clear_error();
  NTG_CHECK_ARG(p && dtx_d && x_d && dir >= 0 && dir <= 2, "ntg_cdtp: bad argument");
  NTG_TRY(need_metrics(p));
  return dv::dispatch<3>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 3>;
    NTG_TRY(fx::use_smem<dv::k_cdtp<LX>>(S::SMEM));
    dv::k_cdtp<LX><<<dv::fx_grid<LX, 3>(p), S::NT, S::SMEM, p->stream>>>(
        dtx_d, x_d, dir, p->nelv, dv::dmat<LX>(p), fx::plan_mats<LX>(p, 1.0), p->met, p->n);
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

int ntg_conv1(ntg_plan* p, double* du_d, const double* u_d, const double* vx_d, const double* vy_d,
              const double* vz_d) {
  clear_error();
  NTG_CHECK_ARG(p && du_d && u_d && vx_d && vy_d && vz_d, "ntg_conv1: null argument");
  NTG_TRY(need_metrics(p));
  return dv::dispatch<2>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 4>;
    NTG_TRY(fx::use_smem<dv::k_conv<LX>>(S::SMEM));
    dv::k_conv<LX><<<dv::fx_grid<LX, 4>(p), S::NT, S::SMEM, p->stream>>>(
        du_d, u_d, vx_d, vy_d, vz_d, p->nelv, fx::plan_mats<LX>(p, 1.0), p->met, p->n);
    NTG_COUNT_LAUNCH();
    NTG_CUDA_TRY(cudaGetLastError());
    return NTG_OK;
  });
}

int ntg_curl(ntg_plan* p, double* w1_d, double* w2_d, double* w3_d, const double* u1_d, const double* u2_d,
             const double* u3_d) {
  clear_error();
  NTG_CHECK_ARG(p && w1_d && w2_d && w3_d && u1_d && u2_d && u3_d, "ntg_curl: null argument");
  NTG_TRY(need_metrics(p));
  return curl_avg(p, w1_d, w2_d, w3_d, u1_d, u2_d, u3_d);
}

int ntg_adjoint_advection_no_dealias(ntg_plan* p, double* fx, double* fy, double* fz, const double* vx,
                                     const double* vy, const double* vz, const double* vxb, const double* vyb,
                                     const double* vzb) {
  clear_error();
  NTG_CHECK_ARG(p && fx && fy && fz && vx && vy && vz && vxb && vyb && vzb,
                "ntg_adjoint_advection_no_dealias: null argument");
  NTG_TRY(need_metrics(p));
  const double* u[3] = {vx, vy, vz};
  const double* ub[3] = {vxb, vyb, vzb};
  double* f[3] = {fx, fy, fz};
  cudaStream_t s = p->stream;
  // f_i -= sum_j u_j opgrad_i(Ub_j) + sum_d cdtp_d(u_i Ub_d), one element pass
  NTG_TRY(dv::dispatch<6>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 9>;
    NTG_TRY(fx::use_smem<dv::k_adv_adj_nd<LX>>(S::SMEM));
    dv::k_adv_adj_nd<LX><<<dv::fx_grid<LX, 9>(p), S::NT, S::SMEM, s>>>(
        f[0], f[1], f[2], u[0], u[1], u[2], ub[0], ub[1], ub[2], p->nelv, dv::dmat<LX>(p),
        fx::plan_mats<LX>(p, 1.0, true), p->met, p->n);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  }));
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

int ntg_linear_advection_no_dealias(ntg_plan* p, double* fx, double* fy, double* fz, const double* vx,
                                    const double* vy, const double* vz, const double* vxb, const double* vyb,
                                    const double* vzb) {
  clear_error();
  NTG_CHECK_ARG(p && fx && fy && fz && vx && vy && vz && vxb && vyb && vzb,
                "ntg_linear_advection_no_dealias: null argument");
  NTG_TRY(need_metrics(p));
  const double* u[3] = {vx, vy, vz};
  const double* ub[3] = {vxb, vyb, vzb};
  double* f[3] = {fx, fy, fz};
  // f_i -= B conv1(u_i; Ub) + B conv1(Ub_i; u), one element pass
  NTG_TRY(dv::dispatch<6>(p->lx, [&](auto L) -> int {
    constexpr int LX = decltype(L)::value;
    using S = dv::FxShape<LX, 9>;
    NTG_TRY(fx::use_smem<dv::k_adv_lin_nd<LX>>(S::SMEM));
    dv::k_adv_lin_nd<LX><<<dv::fx_grid<LX, 9>(p), S::NT, S::SMEM, p->stream>>>(
        f[0], f[1], f[2], u[0], u[1], u[2], ub[0], ub[1], ub[2], p->nelv, dv::dmat<LX>(p),
        fx::plan_mats<LX>(p, 1.0), p->met, p->n);
    NTG_COUNT_LAUNCH();
    return NTG_OK;
  }));
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

int ntg_adjoint_min_dissipation(ntg_plan* p, double* fx, double* fy, double* fz, const double* u, const double* v,
                                const double* w, double scale, const int32_t* zone_d, int64_t nzone, int base) {
  clear_error();
  NTG_CHECK_ARG(p && fx && fy && fz && u && v && w && (nzone == 0 || zone_d) && nzone >= 0,
                "ntg_adjoint_min_dissipation: bad argument");
  NTG_TRY(need_metrics(p));
  const int64_t n = p->n;
  double* t = plan_scratch(p, 6 * n);
  if (!t) return NTG_ERR_ALLOC;
  // the first curl's Binv is applied where the second reads it, the second's where it is added
  NTG_TRY(curl_gs(p, t, t + n, t + 2 * n, u, v, w, nullptr));
  NTG_TRY(curl_gs(p, t + 3 * n, t + 4 * n, t + 5 * n, t, t + n, t + 2 * n, p->binv));
  dv::k_add_zone<<<grid_for(nzone ? nzone : n, 256), 256, 0, p->stream>>>(
      fx, fy, fz, t + 3 * n, t + 4 * n, t + 5 * n, p->binv, scale, nzone ? zone_d : nullptr, nzone, base, n);
  NTG_COUNT_LAUNCH();
  NTG_CUDA_TRY(cudaGetLastError());
  return NTG_OK;
}

}  // extern "C"
