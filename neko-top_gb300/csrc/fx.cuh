// One-dimensional operator applications y = M x on FP64 lines, evaluated in
// 64-bit fixed point on the integer pipes.
//
// What bounds it: an SM retires 2 FP64 instructions per clock (FMA, add and
// the conversion instructions alike) but 64 IMAD.WIDE (32 x 32 + 64 bits), 64
// logic / shift and 128 integer additions (measured: 4.1 against 129 lane
// operations per ns and SM).  A contraction of FP64 lines is therefore integer
// arithmetic here, and to_fix and from_fix use integer and FP32 instructions
// alone, so that the FP64 pipe has only the products around the contractions:
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
// Error: a line's entries keep 60 bits under its largest; products of the low
// limbs are dropped, the middle ones rounded, and the sum is rounded to FP64.
// In units of the row's largest entry times the line's largest, over 200
// thousand uniform lines of every order (D and D^T): at most 2^-52 (lx 2) to
// 2^-51.1 (lx 10), root mean square 2^-54.7 to 2^-54.3.  FP64 FMAs: 2^-52 to
// 2^-49.6, and 2^-54.7 to 2^-53.1.  Each line has its own exponent, so a small
// line beside a large one loses nothing; each row of the matrix has its own
// scale down to a quarter of the largest row's, so the innermost rows, an
// eighth of the end rows at lx = 8, lose a bit of the 60.
//
// Lines whose largest entry is outside [2^-913, 2^977] (NaN and infinity
// included) take the plain FP64 sum instead: same results as without fixed
// point.  A derivative matrix has zeros on its inner diagonal, so where one
// inner entry of a line exceeds all others the sum at its node is one of small
// entries, which integers scaled by the large one have too few bits for.  There
// that sum, or the line's, is taken in FP64 (`guard`, dominated()), so that
// every result is as good as an FP64 sum of its own terms.
#pragma once
#include <stdint.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <mutex>
#include <new>

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
  // every row is scaled to 60 bits by itself (the rows of a derivative matrix
  // differ by a factor of ten): y_A = Y_A 2^(E + k[A] - 1023); the common
  // scale of line_int is kc, Y_A 2^s[A] under it
  int k[RO], s[RO], kc;
};

// host: M row-major (NOUT x NIN), centro-symmetric or -antisymmetric
template <int NIN, int NOUT, typename T0>
Mat<NIN, NOUT> make_mat(const T0* M) {
  using T = Mat<NIN, NOUT>;
  T r;
  long double e[T::RO][T::HE], o[T::RO][T::HO];
  int ex[T::RO], top = -100000;
  for (int A = 0; A < T::RO; ++A) {
    long double mx = 0;
    for (int a = 0; a < T::HE; ++a) {
      const int b = NIN - 1 - a;
      const long double p = M[A * NIN + a], q = M[A * NIN + b];
      e[A][a] = a == b ? p : 0.5L * (p + q);
      mx = std::max(mx, std::fabs(e[A][a]));
      if (a < T::HO) {
        o[A][a] = 0.5L * (p - q);
        mx = std::max(mx, std::fabs(o[A][a]));
      }
    }
    ex[A] = -100000;
    if (mx > 0) std::frexp(mx, &ex[A]);  // mx in [2^(ex-1), 2^ex)
    top = std::max(top, ex[A]);
  }
  if (top == -100000) top = 0;
  // a row's result under the common scale, and the sum of three of them, stay
  // inside 63 bits: |Y_A| <= 2^(XB - 4) sum |M_Aa| / 2^ex, and sum |M_Aa| < 8 2^ex here
  constexpr int LEFT = 63 - 2 - 3 - (T::XB - 4);
  static_assert(LEFT >= 2, "bits");
  for (int A = 0; A < T::RO; ++A) {
    ex[A] = std::max(ex[A], top - LEFT);
    const int sh = 60 - ex[A];
    auto put = [&](long double v, int& h, int& l) {
      const int64_t q = (int64_t)std::llrint(std::ldexp(v, sh));
      l = (int32_t)(uint32_t)(q & 0xffffffffll);
      h = (int32_t)((q - (int64_t)l) >> 32);
    };
    for (int a = 0; a < T::HE; ++a) put(e[A][a], r.eh[A][a], r.el[A][a]);
    for (int a = 0; a < T::HO; ++a) put(o[A][a], r.oh[A][a], r.ol[A][a]);
    r.k[A] = 64 - sh - T::XB + 1;
  }
  r.kc = 64 - (60 - top) - T::XB + 1 - LEFT;
  for (int A = 0; A < T::RO; ++A) r.s[A] = r.k[A] - r.kc;
  return r;
}

// the derivative matrix of the GLL points, its transpose times `scale`, and
// both as FP64 numbers
template <int LX>
struct Mats {
  Mat<LX, LX> D, DT;
  double d[LX * LX], dt[LX * LX];
};

// w: null, or weights for the form of D^T that acts before them:
// DT = W^-1 D^T W, so that D^T (W f) = W (DT f)
template <int LX>
Mats<LX> make_mats(const double* D, const double* w, double scale) {
  Mats<LX> P;
  long double t[LX * LX];
  for (int i = 0; i < LX; ++i)
    for (int j = 0; j < LX; ++j) {
      t[i * LX + j] = (long double)D[j * LX + i] * scale;
      if (w) t[i * LX + j] = t[i * LX + j] * w[j] / w[i];
      P.d[i * LX + j] = D[i * LX + j];
      P.dt[i * LX + j] = (double)t[i * LX + j];
    }
  P.D = make_mat<LX, LX>(D);
  P.DT = make_mat<LX, LX>(t);
  return P;
}

// The plan's matrices, made once per plan and scale (a constant h1 or mu).
// The few scales in use at a time stay; a copy goes to the caller, so plans
// may be used from several threads.
// `weighted`: the D^T that acts before the GLL weights (make_mats).
template <int LX>
Mats<LX> plan_mats(const ntg_plan* p, double scale, bool weighted = false) {
  std::lock_guard<std::mutex> lk(p->fx->mu);
  auto& c = p->fx->mats;
  for (auto& e : c)
    if (e.scale == scale && e.weighted == weighted) return *static_cast<const Mats<LX>*>(e.mats.get());
  const Mats<LX> m = make_mats<LX>(p->D, weighted ? p->wq : nullptr, scale);
  try {
    if (c.size() >= 6) c.erase(c.begin());
    c.push_back({scale, weighted, std::make_shared<Mats<LX>>(m)});
  } catch (const std::bad_alloc&) {  // not kept, then: no exception leaves the C entry points
  }
  return m;
}

// whether a constant factor may be folded into a matrix (its exponent offset must stay small)
inline bool foldable(double c) { return c == 0.0 || (std::fabs(c) > 1e-6 && std::fabs(c) < 1e6); }

// lets Kernel use `bytes` of dynamic shared memory and the largest carve-out; set once per device
template <auto Kernel>
int use_smem(size_t bytes) {
  static std::atomic<uint64_t> set{0};
  int dev = 0;
  NTG_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (set.load(std::memory_order_acquire) & bit) return NTG_OK;
  NTG_CUDA_TRY(cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  NTG_CUDA_TRY(cudaFuncSetAttribute(Kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared));
  set.fetch_or(bit, std::memory_order_release);
  return NTG_OK;
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

// Whether one inner entry of a line held under the exponent E exceeds all
// others by three binary orders or more.  In 60 thousand lines of each kind
// (normal, 10^-2 to 1, 10^-6 to 1, one outlier of up to 2^30; lx 3 to 10) the
// sums' root mean square errors, over the sums of their terms' absolute
// values, were 0.5 to 1.2 times those of FP64 FMAs with such lines summed in
// FP64; without, they grow with the outlier.  One normal line in 2500 is such a
// line at lx = 8, one in 95 at lx = 4.
template <int N>
__device__ __forceinline__ bool dominated(const double (&x)[N], int E) {
  int t = 0;
#pragma unroll
  for (int l = 0; l < N; ++l) {
    const int near = (E - 3 - ((__double2hiint(x[l]) >> 20) & 0x7ff)) >> 31;  // -1: within two orders of the largest
    t += l == 0 || l == N - 1 ? 2 * near : near;
  }
  return t == -1;
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

// Y = M X for a line of integers; out(A, row, Y_A) per output, row = the
// one of the mirrored rows A, NOUT-1-A whose scale holds
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
      out(A, A, ANTI ? dot_limbs<T::HO>(M.oh[A], M.ol[A], oh, ol) : dot_limbs<T::HE>(M.eh[A], M.el[A], eh, el));
    } else {
      const int64_t p = dot_limbs<T::HE>(M.eh[A], M.el[A], eh, el), q = dot_limbs<T::HO>(M.oh[A], M.ol[A], oh, ol);
      out(A, A, p + q);
      out(B, A, ANTI ? q - p : p - q);
    }
  }
}

// M x of an FP64 line as integers: out(A, Y_A), the result being
// Y 2^(K - 1023) with K returned; K = kZero: zeros; K = kSlow: FP64 numbers in
// the integers' bits.  Md is the plain matrix (row-major, times the same
// scale) of the FP64 sums; get(A) returns what out took.  guard: the node of a
// dominant entry gets its FP64 sum, which waits in local memory meanwhile (in
// registers the kernels spilled more, 0.2 KB a thread at lx = 8).
template <int NIN, int NOUT, bool ANTI, typename F, typename G>
__device__ __forceinline__ int line_int(const Mat<NIN, NOUT>& M, const double* Md, const double (&x)[NIN], bool guard,
                                        F&& out, G&& get) {
  const int E = line_exp<NIN>(x);
  if (E >= 0 && E != kSlow) {
    volatile double own;
    volatile int at;
    bool dom = false;
    if constexpr (NIN > 2) {
      dom = guard && dominated<NIN>(x, E);
      if (dom) {
        int i = 1;
#pragma unroll
        for (int l = 2; l < NIN - 1; ++l)
          if (((__double2hiint(x[l]) >> 20) & 0x7ff) == E) i = l;
        double acc = 0.0;
#pragma unroll
        for (int l = 0; l < NIN; ++l) acc = fma(Md[i * NIN + l], x[l], acc);
        own = acc;
        at = i;
      }
    }
    int64_t X[NIN];
#pragma unroll
    for (int l = 0; l < NIN; ++l) X[l] = to_fix<Mat<NIN, NOUT>::XB>(x[l], E);
    line<NIN, NOUT, ANTI>(M, X, [&](int A, int row, int64_t Y) { out(A, shl(Y, M.s[row])); });
    const int K = E + M.kc;
    if (!dom) return K;
    const int i = at;
    const double acc = own;
#pragma unroll
    for (int A = 0; A < NOUT; ++A) out(A, (int64_t)__double_as_longlong(A == i ? acc : from_fix(get(A), K)));
    return kSlow;
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

// M x of an FP64 line as FP64 numbers: out(A, y_A).  guard: lines with a
// dominant entry as FP64 sums
template <int NIN, int NOUT, bool ANTI, typename F>
__device__ __forceinline__ void line_dbl(const Mat<NIN, NOUT>& M, const double* Md, const double (&x)[NIN], bool guard,
                                         F&& out) {
  int E = line_exp<NIN>(x);
  if constexpr (NIN > 2)
    if (guard && E >= 0 && E != kSlow && dominated<NIN>(x, E)) E = kSlow;
  if (E >= 0 && E != kSlow) {
    int64_t X[NIN];
#pragma unroll
    for (int l = 0; l < NIN; ++l) X[l] = to_fix<Mat<NIN, NOUT>::XB>(x[l], E);
    line<NIN, NOUT, ANTI>(M, X, [&](int A, int row, int64_t Y) { out(A, from_fix(Y, E + M.k[row])); });
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

// line_int into y, entries `st` apart
template <int NIN, int NOUT, bool ANTI>
__device__ __forceinline__ int line_int_to(const Mat<NIN, NOUT>& M, const double* Md, const double (&x)[NIN], bool guard,
                                           double* y, int st) {
  return line_int<NIN, NOUT, ANTI>(
      M, Md, x, guard, [&](int A, int64_t v) { y[A * st] = __longlong_as_double(v); },
      [&](int A) { return (int64_t)__double_as_longlong(y[A * st]); });
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

// A tile of L^3 FP64 numbers in shared memory with an odd row stride: the
// lines of all three directions are read and written without bank conflicts.
template <int L>
struct Tile {
  static constexpr int L2 = L * L, L3 = L2 * L, RS = L | 1, SIZE = L2 * RS;
  static __device__ __forceinline__ int at(int node) { return node / L * RS + node % L; }
  // first entry and stride of line q (0 .. L2-1) of direction d
  static __device__ __forceinline__ int base(int d, int q) {
    const int p = q % L, r = q / L;
    return d == 0 ? (p + L * r) * RS : d == 1 ? L * r * RS + p : r * RS + p;
  }
  static __device__ __forceinline__ int stride(int d) { return d == 0 ? 1 : d == 1 ? RS : L * RS; }
};

// the derivative tile of direction d of `in`, line q, into `out` (which may be
// `in`).  guard: the derivatives themselves are results, not the start of
// fluxes along the same lines (whose own sums then have the large terms)
template <int L>
__device__ __forceinline__ void deriv_line(const Mat<L, L>& D, const double* d_, const double* in, double* out, int d,
                                           int q, bool guard = true) {
  const int b = Tile<L>::base(d, q), st = Tile<L>::stride(d);
  double x[L];
#pragma unroll
  for (int l = 0; l < L; ++l) x[l] = in[b + l * st];
  line_dbl<L, L, true>(D, d_, x, guard, [&](int A, double y) { out[b + A * st] = y; });
}

// The transposed derivative of a flux tile in place, as integers; *k: their
// exponent.  guard: unless the fluxes are a gradient times metrics and
// constants.  A node whose flux exceeds its lines' others in all three
// directions is one of a coefficient or a velocity, not of a gradient.
template <int L>
__device__ __forceinline__ void flux_line(const Mat<L, L>& DT, const double* dt_, double* f, int* k, int d, int q,
                                          bool guard = true) {
  const int b = Tile<L>::base(d, q), st = Tile<L>::stride(d);
  double x[L];
#pragma unroll
  for (int l = 0; l < L; ++l) x[l] = f[b + l * st];
  *k = line_int_to<L, L, true>(DT, dt_, x, guard, f + b, st);
}

// the sum of the three transposed derivatives at a node: f[d], k[d] (k + d L2) of flux_line
template <int L>
__device__ __forceinline__ double flux_sum(const double* f0, const double* f1, const double* f2, const int* k, int node) {
  constexpr int L2 = L * L;
  const int i = node % L, j = node / L % L, kk = node / L2, p = Tile<L>::at(node);
  return sum3(__double_as_longlong(f0[p]), k[j + L * kk], __double_as_longlong(f1[p]), k[L2 + i + L * kk],
              __double_as_longlong(f2[p]), k[2 * L2 + i + L * j]);
}

}  // namespace fx
}  // namespace ntg
