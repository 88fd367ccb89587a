// One-dimensional operator applications y = M x on FP64 lines, evaluated in
// 64-bit fixed point on the integer pipes.
//
// What bounds it: an SM retires 2 FP64 instructions per clock (FMA, add and
// every conversion to or from FP64 alike) but 64 IMAD.WIDE (32 x 32 + 64
// bits), 64 logic / shift and 128 integer additions (measured: 4.1 against
// 129 lane operations per ns and SM).  A contraction of FP64 lines is
// therefore exact integer arithmetic here:
//
//   to_fix    the line's values become 60-bit integers under the exponent
//             of its largest entry;
//   line      the matrix, split into its parts even and odd about the
//             centre (all of the operators on symmetric point sets are
//             centro-symmetric or -antisymmetric), stands in the kernel
//             parameters as two signed 32-bit limbs per entry; three
//             IMAD.WIDE per product (high x high, and both cross products),
//             half as many products as the full matrix has;
//   from_fix  the 64-bit sum becomes an FP64 number, rounded to nearest.
//
// Error: products of the low limbs (2^-60 of the largest matrix entry times
// the largest line entry) and the last bit of the sum (2^-57) are dropped,
// which is below the rounding of the eight FP64 FMAs it replaces; each line
// has its own exponent, so a small line beside a large one loses nothing.
//
// Lines whose largest entry is outside [2^-913, 2^977] (NaN and infinity
// included) take the plain FP64 sum instead (`ok` false): same results as
// without fixed point.
#pragma once
#include <stdint.h>
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace ntg {
namespace fx {

constexpr int kZero = -4096;      // exponent of a line of zeros
constexpr int kSlow = 0x40000000; // exponent mark of a line held as FP64 numbers

// the matrix M (NOUT x NIN) = round(M 2^sh), limbs h 2^32 + l of its even
// and odd parts: even input e_a = x_a + x_(NIN-1-a) (the middle entry
// itself), odd input o_a = x_a - x_(NIN-1-a)
template <int NIN, int NOUT>
struct Mat {
  static constexpr int HE = (NIN + 1) / 2, HO = NIN / 2, RO = (NOUT + 1) / 2;
  // bits of the line integers: sums of HE products of both limbs stay inside 63 bits
  static constexpr int XB = HE <= 5 ? 60 : 59;
  int eh[RO][HE], el[RO][HE], oh[RO][HO], ol[RO][HO];
  int k0;  // exponent offset of the result: y = Y 2^(E + k0 - 1023)
};

// host: M row-major (NOUT x NIN), centro-symmetric (+1) or -antisymmetric, times scale
template <int NIN, int NOUT>
Mat<NIN, NOUT> make_mat(const double* M, double scale = 1.0) {
  using T = Mat<NIN, NOUT>;
  T r;
  long double e[T::RO][T::HE], o[T::RO][T::HO], mx = 0;
  for (int A = 0; A < T::RO; ++A) {
    for (int a = 0; a < T::HE; ++a) {
      const int b = NIN - 1 - a;
      const long double p = (long double)M[A * NIN + a] * scale, q = (long double)M[A * NIN + b] * scale;
      e[A][a] = a == b ? p : 0.5L * (p + q);
      if (a < T::HO) o[A][a] = 0.5L * (p - q);
      mx = std::max(mx, std::fabs(e[A][a]));
      if (a < T::HO) mx = std::max(mx, std::fabs(o[A][a]));
    }
  }
  int ex = 0;
  if (mx > 0) std::frexp(mx, &ex);  // mx in [2^(ex-1), 2^ex)
  const int sh = 60 - ex;
  auto put = [&](long double v, int& h, int& l) {
    const int64_t q = (int64_t)std::llrint(std::ldexp(v, sh));
    l = (int32_t)(uint32_t)(q & 0xffffffffll);
    h = (int32_t)((q - (int64_t)l) >> 32);
  };
  for (int A = 0; A < T::RO; ++A) {
    for (int a = 0; a < T::HE; ++a) put(e[A][a], r.eh[A][a], r.el[A][a]);
    for (int a = 0; a < T::HO; ++a) put(o[A][a], r.oh[A][a], r.ol[A][a]);
  }
  r.k0 = 64 - sh - T::XB + 1;
  return r;
}

__device__ __forceinline__ int64_t mk64(uint32_t lo, uint32_t hi) {
  int64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void sp64(int64_t v, uint32_t& lo, uint32_t& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ int64_t sar(int64_t v, int s) {  // shift counts past 63 give the sign
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}
__device__ __forceinline__ int64_t shl(int64_t v, int s) {  // past 63: 0
  int64_t r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}

// the exponent the line x is held under: the biased exponent of its largest
// entry, kZero for zeros, kSlow when it must stay in FP64
template <int N>
__device__ __forceinline__ int line_exp(const double (&x)[N]) {
  int m = 0;
#pragma unroll
  for (int l = 0; l < N; ++l) m = max(m, __double2hiint(x[l]) & 0x7fffffff);
  const int E = m >> 20;
  if (E >= 110 && E <= 2000) return E;
  int any = m;
#pragma unroll
  for (int l = 0; l < N; ++l) any |= __double2loint(x[l]);
  return any ? kSlow : kZero;
}

// x as an integer of XB bits under the exponent E
template <int XB>
__device__ __forceinline__ int64_t to_fix(double x, int E) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int e = (hi >> 20) & 0x7ff, s = hi >> 31;
  const uint32_t mh = ((uint32_t)hi & 0xfffffu) | 0x100000u;
  const uint32_t th = __funnelshift_l((uint32_t)lo, mh, 10) ^ (uint32_t)s, tl = ((uint32_t)lo << 10) ^ (uint32_t)s;
  return sar(mk64(tl, th), E - e + (63 - XB));
}

// Y 2^(K - 1023) as an FP64 number, rounded to nearest; |Y| < 2^63
__device__ __forceinline__ double from_fix(int64_t Y, int K) {
  uint32_t lo, hi;
  const int64_t sg = Y >> 63;
  const int64_t A = (Y ^ sg) - sg;
  sp64(A, lo, hi);
  // the leading bit's position from an FP32 conversion that rounds towards zero
  const int ef = __float_as_int(__fmaf_rz(__uint2float_rz(hi), 4294967296.f, __uint2float_rz(lo))) >> 23;  // 127 + p
  const int64_t m = (int64_t)((uint64_t)(shl(A, 189 - ef) + 512) >> 10);  // in [2^52, 2^53]
  sp64(m, lo, hi);
  hi += (uint32_t)(K + ef - 128) << 20;
  hi = ef ? hi : 0u;
  hi |= (uint32_t)(sg >> 32) & 0x80000000u;
  return __hiloint2double((int)hi, (int)lo);
}

// sum of NT products, each of two limbs, without the low x low ones
template <int NT>
__device__ __forceinline__ int64_t dot_limbs(const int (&mh)[NT], const int (&ml)[NT], const int (&xh)[NT],
                                             const int (&xl)[NT]) {
  int64_t hh = 0, mid = 0x80000000ll;
#pragma unroll
  for (int a = 0; a < NT; ++a) {
    hh += (int64_t)mh[a] * xh[a];
    mid += (int64_t)mh[a] * xl[a];
    mid += (int64_t)ml[a] * xh[a];
  }
  return hh + (mid >> 32);
}

// Y = M X for a line of integers; out(A, Y_A) per output
template <int NIN, int NOUT, bool ANTI, typename F>
__device__ __forceinline__ void line(const Mat<NIN, NOUT>& M, const int64_t (&X)[NIN], F&& out) {
  using T = Mat<NIN, NOUT>;
  int eh[T::HE], el[T::HE], oh[T::HO], ol[T::HO];
#pragma unroll
  for (int a = 0; a < T::HE; ++a) {
    const int b = NIN - 1 - a;
    uint32_t l, h;
    sp64(a == b ? X[a] : X[a] + X[b], l, h);
    el[a] = (int)l;
    eh[a] = (int)(h + (l >> 31));
    if (a < T::HO) {
      sp64(X[a] - X[b], l, h);
      ol[a] = (int)l;
      oh[a] = (int)(h + (l >> 31));
    }
  }
#pragma unroll
  for (int A = 0; A < T::RO; ++A) {
    const int B = NOUT - 1 - A;
    if (A == B) {
      out(A, ANTI ? dot_limbs<T::HO>(M.oh[A], M.ol[A], oh, ol) : dot_limbs<T::HE>(M.eh[A], M.el[A], eh, el));
    } else {
      const int64_t p = dot_limbs<T::HE>(M.eh[A], M.el[A], eh, el), q = dot_limbs<T::HO>(M.oh[A], M.ol[A], oh, ol);
      out(A, p + q);
      out(B, ANTI ? q - p : p - q);
    }
  }
}

// M x of an FP64 line as integers: out(A, Y_A), the result being
// Y 2^(K - 1023) with K returned; K = kZero: zeros; K = kSlow: the FP64 sums
// themselves, in the integers' bits.  Md is the plain matrix (row-major,
// times the same scale) of the FP64 sums.
template <int NIN, int NOUT, bool ANTI, typename F>
__device__ __forceinline__ int line_int(const Mat<NIN, NOUT>& M, const double* Md, const double (&x)[NIN], F&& out) {
  const int E = line_exp<NIN>(x);
  if (E >= 0 && E != kSlow) {
    int64_t X[NIN];
#pragma unroll
    for (int l = 0; l < NIN; ++l) X[l] = to_fix<Mat<NIN, NOUT>::XB>(x[l], E);
    line<NIN, NOUT, ANTI>(M, X, out);
    return E + M.k0;
  }
#pragma unroll
  for (int A = 0; A < NOUT; ++A) {
    double acc = 0.0;
    if (E == kSlow) {
#pragma unroll
      for (int l = 0; l < NIN; ++l) acc = fma(Md[A * NIN + l], x[l], acc);
    }
    out(A, (int64_t)__double_as_longlong(acc));
  }
  return E;
}

// M x of an FP64 line as FP64 numbers: out(A, y_A)
template <int NIN, int NOUT, bool ANTI, typename F>
__device__ __forceinline__ void line_dbl(const Mat<NIN, NOUT>& M, const double* Md, const double (&x)[NIN], F&& out) {
  const int E = line_exp<NIN>(x);
  if (E >= 0 && E != kSlow) {
    int64_t X[NIN];
#pragma unroll
    for (int l = 0; l < NIN; ++l) X[l] = to_fix<Mat<NIN, NOUT>::XB>(x[l], E);
    const int K = E + M.k0;
    line<NIN, NOUT, ANTI>(M, X, [&](int A, int64_t Y) { out(A, from_fix(Y, K)); });
    return;
  }
#pragma unroll
  for (int A = 0; A < NOUT; ++A) {
    double acc = 0.0;
    if (E == kSlow) {
#pragma unroll
      for (int l = 0; l < NIN; ++l) acc = fma(Md[A * NIN + l], x[l], acc);
    }
    out(A, acc);
  }
}

// the sum of three results of line_int
__device__ __forceinline__ double sum3(int64_t a, int Ka, int64_t b, int Kb, int64_t c, int Kc) {
  const int K = max(Ka, max(Kb, Kc));
  if (K != kSlow) return from_fix(sar(a, K - Ka) + sar(b, K - Kb) + sar(c, K - Kc), K);
  const double x = Ka == kSlow ? __longlong_as_double(a) : from_fix(a, Ka);
  const double y = Kb == kSlow ? __longlong_as_double(b) : from_fix(b, Kb);
  const double z = Kc == kSlow ? __longlong_as_double(c) : from_fix(c, Kc);
  return x + y + z;
}

}  // namespace fx
}  // namespace ntg
