// FP64 sums of products on the integer units.
//
// GB300 issues one FP64 instruction (multiply-add, add, compare, minimum alike) per 19 cycles
// and SM, but a 32 x 32 + 64 bit integer multiply-add every half cycle (both measured, all warps
// resident).  The FP64 stage kernels were bound by their sums of products with per-element or
// constant matrices, so those run in fixed point: the factors of a sum are scaled by powers of two
// to 60-bit integers, each kept as two signed digits x = h 2^31 + l.  A product is three of its four
// digit products (the low one is below 2^-59 of the scale), accumulated without rounding in two
// 64-bit words: about 1.5 cycles instead of 19.  Everything that is not a sum of products (the
// Runge-Kutta update, the limiter's means, differences and division) stays in FP64, whose pipe runs
// beside the integer units.
//
// Error.  Of a sum of n products, the matrix row scaled by its sum of magnitudes |a| and the vector by
// its largest magnitude |x|: the digits of a are rounded (2^-61 |a| each), those of x cut off (2^-60 |x|),
// the low products left out (2^-59 each), together at most (2.5 n + 1) 2^-60 |a| |x| and about 2^-60 |a| |x| in
// the mean, where an FP64 chain is off by up to n 2^-53 sum |a_j x_j|.  So that |a| |x| stays near sum |a_j x_j|,
// what differs in size by nature has a scale of its own: every row of a matrix, every edge's velocity,
// the element and each of its neighbours, the mean and the rest of the coefficients, the derivatives of
// different order.  tests/test_fixed_point_cpu.py compares both forms with 80-bit sums, coefficient by
// coefficient.  An element with exponents outside the ranges below, or that holds an infinity or a NaN, is
// left to the FP64 form of the same terms.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "dgadv_kernels.cuh"

namespace dgadv {

// The constant tables of a degree in digits: defined by the FP64 unit.
template <int P> __device__ __forceinline__ const FxTab<P> &fx_tab();

namespace fx {

constexpr int kW = 60;                       // bits of a scaled factor
constexpr int kD = 31;                       // bits of the low digit
// biased exponents taken: matrices 2^-200 .. 2^400, vectors 2^-700 .. 2^400 (a solution's far tail
// runs through small numbers); products and their units stay normal
constexpr int kMatLo = 823, kExpLo = 323, kExpHi = 1423;

__device__ __forceinline__ int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// |x| in units of 2^(E - 1022 - W), truncated: |x| < 2^(E - 1022) for expo(x) <= E, so the result is
// below 2^W.  Zeros and denormals (expo 0) shift out to zero for E >= 64.
template <int W> __device__ __forceinline__ unsigned long long fix_mag(double x, int E) {
  const unsigned long long m = ((unsigned long long)__double_as_longlong(x) & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL;
  return (m << (W - 53)) >> min(E - expo(x), 63);
}
template <int W> __device__ __forceinline__ long long fix(double x, int E) {
  const long long v = (long long)fix_mag<W>(x, E), sg = (long long)(__double2hiint(x) >> 31);
  return (v ^ sg) - sg;
}
// x in the same units to the nearest (halves up).
template <int W> __device__ __forceinline__ long long fix_near(double x, int E) { return (fix<W + 1>(x, E) + 1) >> 1; }
// X = h 2^31 + l, -2^30 <= l < 2^30
__host__ __device__ __forceinline__ Dig digits(long long X) {
  Dig d;
  d.l = (int)((unsigned)X << 1) >> 1;
  d.h = (int)((X - d.l) >> kD);
  return d;
}
// The digits of x in units of 2^(E - 1022 - kW): both of the sign of x, |l| < 2^31, |h| < 2^29.
__device__ __forceinline__ Dig digits_of(double x, int E) {
  const unsigned long long v = fix_mag<kW>(x, E);
  const int sg = __double2hiint(x) >> 31;
  Dig d;
  d.l = ((int)((unsigned)v & 0x7fffffffu) ^ sg) - sg;
  d.h = ((int)(v >> kD) ^ sg) - sg;
  return d;
}
// The digits of a matrix entry below 2^(E - 1022), to the nearest.
__host__ __device__ __forceinline__ Dig digits_near(double x, int E) {
  return digits((long long)rint(ldexp(x, kW + 1022 - E)));
}
// V as a double, to the nearest: two FP64 additions of the words' bit patterns, 2^84 + 2^63 + hi 2^32
// and 2^52 + lo.
__device__ __forceinline__ double to_double(long long V) {
  const double hi = __hiloint2double(0x45300000, (int)(V >> 32) ^ (int)0x80000000);
  const double lo = __hiloint2double(0x43300000, (int)V);
  return (hi - (0x1p84 + 0x1p63 + 0x1p52)) + lo;
}
// V 2^u in integers (round half up in the magnitude), where FP64 additions are dearer; the
// caller's exponents keep it normal.
__device__ __forceinline__ double to_double_int(long long V, int u) {
  if (V == 0) return 0.0;
  const unsigned long long mag = V < 0 ? 0ULL - (unsigned long long)V : (unsigned long long)V;
  const int lz = __clzll((long long)mag);
  const unsigned long long m = ((mag << lz) >> 10) + 1;
  const unsigned long long b = ((unsigned long long)(1023 + 62 - lz + u) << 52) + (m >> 1);
  return __longlong_as_double((long long)(b | ((unsigned long long)V & 0x8000000000000000ULL)));
}
__device__ __forceinline__ double to_double(long long V, int u) {   // V 2^u
  const double d = to_double(V);
  return V == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (u << 20), __double2loint(d));
}
// The largest exponent E among x[0 .. n); false where they are left to FP64: outside the range, or a
// denormal among nothing larger.  All zero: E = 0.
template <int n> __device__ __forceinline__ bool scale_of(const double *x, int &E) {
  int e = 0;
#pragma unroll
  for (int j = 0; j < n; ++j) e = max(e, __double2hiint(x[j]) & 0x7fffffff);
  E = e >> 20;
  if (E < kExpLo) {
    int low = 0;
#pragma unroll
    for (int j = 0; j < n; ++j) low |= __double2loint(x[j]);
    return (e | low) == 0;
  }
  return E <= kExpHi;
}

// Running sum: h 2^62 + m 2^31 in units of the factors' product.  In range for up to 12 terms: with one
// factor's |l| <= 2^30 and its magnitudes' sum at most 2^60 (a table or a matrix row), the other
// below 2^60 with |l| < 2^31, |m| stays below 12 2^59 + 2^60.
struct Sum {
  long long h = 0, m = 0;
  __device__ __forceinline__ void add(const Dig &a, const Dig &b) {
    h += (long long)a.h * b.h;
    m += (long long)a.h * b.l;
    m += (long long)a.l * b.h;
  }
  // with the low product too
  __device__ __forceinline__ void add_all(const Dig &a, const Dig &b) {
    add(a, b);
    m += ((long long)a.l * b.l) >> kD;
  }
  // the sum over 2^(31 + S)
  template <int S> __device__ __forceinline__ long long over() const {
    static_assert(S >= 0 && S <= 31, "");
    return (h << (31 - S)) + (m >> S);
  }
};
__device__ __forceinline__ long long shr(long long x, int s) { return x >> min(s, 63); }   // s >= 0

// Exponents of an element's rows: the largest in 11 bits of a word, the others as bytes below it.
// Byte i of the words w (stride Kp).
__device__ __forceinline__ int byte_of(const unsigned *w, int i) { return (int)((w[i >> 2] >> (8 * (i & 3))) & 0xffu); }

// ---------------------------------------------------------------------------------------------
// The element operator's exponents: word 0 holds the largest in bits 0..10, the inflow edges in
// 22..24 and in bit 31 that the element is not in fixed point; then bytes below the largest: N rows'
// entries of each part, 3 edges.  The parts: the mean and the other coefficients.
template <int P> struct OpExp {
  static constexpr int N = Dims<P>::N;
  static constexpr int kParts = op_parts(P), kEdge = kParts * N, kWords = op_exp_words(P) - 1;
  __host__ __device__ static constexpr int begin(int s) { return s == 0 ? 0 : s == 1 ? 1 : N; }
  int head = (int)0x80000000u;
  unsigned w[kWords];
  __device__ __forceinline__ void load(const int *__restrict__ ax, int Kp, int k) {
    head = ax[k];
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = (unsigned)ax[(size_t)(1 + i) * Kp + k];
  }
  __device__ __forceinline__ bool inflow(int n) const { return (head >> (22 + n)) & 1; }
  __device__ __forceinline__ int at(int i) const { return (head & 2047) - byte_of(w, i); }
};

// cDot of one element from its element operator: A c - sum over the inflow edges' points of
// Fphi v trace(neighbour) (stage_op_tile, kOpElement).
//   sA, sV: digits of A (row i N + j) and of v (row n R + r), row stride st
// Returns false (cdot untouched) where the element is left to FP64.
template <int P>
__device__ __forceinline__ bool element_cdot(const FxTab<P> &tb, const Dig *sA, const Dig *sV, int st,
                                             const OpExp<P> &ax, const double *c, const double (*cn)[Dims<P>::N],
                                             int code, double *cdot) {
  constexpr int N = Dims<P>::N, R = Dims<P>::R;
  if (ax.head < 0) return false;
  constexpr int S = OpExp<P>::kParts;
  // scales: every part of the coefficients, every neighbour
  int E[S], En[3] = {0, 0, 0};
  bool ok = scale_of<1>(c, E[0]);
  if constexpr (S > 1) ok = scale_of<N - 1>(c + 1, E[1]) && ok;
#pragma unroll
  for (int n = 0; n < 3; ++n)
    if (ax.inflow(n)) ok = scale_of<N>(cn[n], En[n]) && ok;
  if (!ok) return false;
  // inflow terms: fl[i] below 3 2^60 in units of 2^(xf[i] - 2044 - 60)
  long long fl[N];
  int xf[N];
#pragma unroll
  for (int i = 0; i < N; ++i) { fl[i] = 0; xf[i] = -8192; }
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    if (En[n] == 0) continue;
    const int np = (code >> (2 * n)) & 3;
    long long q[R];
    unsigned long long most = 0;
    {
      Dig d[N];
#pragma unroll
      for (int j = 0; j < N; ++j) d[j] = digits_of(cn[n][j], En[n]);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const Dig v = sV[(size_t)(n * R + r) * st];
        q[r] = 0;
        if (!(v.h < 0 || (v.h == 0 && v.l < 0))) continue;
        Sum tr, vt;
#pragma unroll
        for (int j = 0; j < N; ++j) tr.add(tb.thetaPhi[n][np][r][j], d[j]);
        vt.add_all(digits(tr.over<29>()), v);        // trace below 2^60, unit 2^(En + eT - 60)
        q[r] = -vt.over<29>();
        most = max(most, (unsigned long long)(q[r] < 0 ? ~q[r] : q[r]));
      }
    }
    // the edge's largest flux to 60 bits: the scales of the trace and the velocity are bounds
    const int up = __clzll((long long)most) - 4, ge = En[n] + ax.at(OpExp<P>::kEdge + n) + tb.eT - up;
    if (most == 0) continue;
    Sum f[N];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Dig d = digits(q[r] << up);
#pragma unroll
      for (int i = 0; i < N; ++i) f[i].add(tb.Fphi[n][r][i], d);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int xe = ge + tb.eF[n][i], x = max(xe, xf[i]);
      fl[i] = shr(fl[i], x - xf[i]) + shr(f[i].template over<29>(), x - xe);
      xf[i] = x;
    }
  }
  // every part below 2^60 in units of 2^(x - 60), fl below 3 2^60: added in the coarsest of the units
  Dig d[N];
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int j = OpExp<P>::begin(s); j < OpExp<P>::begin(s + 1); ++j) d[j] = digits_of(c[j], max(E[s], kExpLo));
#pragma unroll
  for (int i = 0; i < N; ++i) {
    long long part[S];
    int xs[S], x = xf[i];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      Sum a;
#pragma unroll
      for (int j = OpExp<P>::begin(s); j < OpExp<P>::begin(s + 1); ++j) a.add(sA[(size_t)(i * N + j) * st], d[j]);
      part[s] = a.template over<29>();
      xs[s] = E[s] ? ax.at(s * N + i) + E[s] : 0;
      x = max(x, xs[s]);
    }
    long long v = shr(fl[i], x - xf[i]);
#pragma unroll
    for (int s = 0; s < S; ++s) v += shr(part[s], x - xs[s]);
    cdot[i] = to_double(v, x - 2044 - 60);
  }
  return true;
}

// ---------------------------------------------------------------------------------------------
// The linear limiter's factor (vertex_alpha_1div): the least of six ratios num / den, the distance to a
// patch extreme over the tolerance plus or minus the slope towards the vertex.  num, a difference of
// means, is one FP64 subtraction; den is exact to 2^-60 of the larger of the slopes and 2^-22, in
// integers.  The least is found by 32-bit keys of the ratios, to 20 bits, and where keys are that close
// from 64-bit mantissas; then one division.
struct Scaled {                  // mantissa with its top bit set, times 2^e
  unsigned long long m;
  int e;
};
__device__ __forceinline__ Scaled normalized(unsigned long long m, int e) {
  const int lz = __clzll((long long)m);
  return Scaled{m << lz, e - lz};
}
__device__ __forceinline__ Scaled times(const Scaled &a, const Scaled &b) {
  const unsigned long long p = __umul64hi(a.m, b.m);   // off by less than 2^-62 of itself
  return (long long)p < 0 ? Scaled{p, a.e + b.e} : Scaled{p << 1, a.e + b.e - 1};
}
__device__ __forceinline__ Scaled mantissa(double x) {   // x > 0, normal
  return normalized(((unsigned long long)__double_as_longlong(x) & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL, expo(x));
}
// num / den < num2 / den2, all positive, the dens in one unit
__device__ __forceinline__ bool ratio_less(double num, long long den, double num2, long long den2) {
  const Scaled a = times(mantissa(num), normalized((unsigned long long)den2, 0));
  const Scaled b = times(mantissa(num2), normalized((unsigned long long)den, 0));
  return a.e < b.e || (a.e == b.e && a.m < b.m);
}
constexpr int kKeyOne = 0x3f800000 >> 3, kKeyClose = 4, kNone = 1 << 30;   // the key of 1; keys are off by at most 2
__device__ __forceinline__ int ratio_key(double num, long long den, int unit) {   // 3 |num| / (|den| 2^unit)
  const float a = __int_as_float(0x3f800000 | ((__double2hiint(num) & 0xfffff) << 3));
  return (__float_as_int(__fdividef(3.0f * a, fabsf(__ll2float_rn(den)))) >> 3) + (int)((unsigned)(expo(num) - 1023 - unit) << 20);
}
// 3 num < den 2^unit
__device__ __forceinline__ bool below_one(double num, long long den, int unit) {
  const unsigned long long f = ((unsigned long long)__double_as_longlong(num) & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL;
  const Scaled a = normalized(3 * f, expo(num) - 1075), b = normalized((unsigned long long)den, unit);
  return a.e < b.e || (a.e == b.e && a.m < b.m);
}

// Returns 0: not limited, 1: limited by alpha, -1: left to FP64.
//   lo, hi: the patch extremes at the vertices, data: boundary values where dmask has the vertex's bit
//   u: the mean and the reference derivatives at the barycentre
__device__ __forceinline__ int linear_alpha(const double lo[3], const double hi[3], int dmask, const double data[3],
                                            const double u[3], double &alpha) {
  int big = max(expo(u[0]), max(expo(u[1]), expo(u[2])));
  double num[3][2];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    double mn = lo[n], mx = hi[n];
    if ((dmask >> n) & 1) {
      mn = fmin(mn, data[n]);
      mx = fmax(mx, data[n]);
      big = max(big, expo(data[n]));
    }
    big = max(big, max(expo(mn), expo(mx)));
    num[n][0] = u[0] - mn;
    num[n][1] = mx - u[0];
  }
  if (big > kExpHi) return -1;
  const int G = max(max(expo(u[1]), expo(u[2])), 1000), unit = G - 1022 - kW;
  const long long U1 = fix<kW>(u[1], G), U2 = fix<kW>(u[2], G), tol3 = 3 * fix<kW>(1.e-8, G);
  const long long dV3[3] = {-(U1 + U2), 2 * U1 - U2, 2 * U2 - U1};
  bool zero = false, past = false, close = false;
  int best = kNone;
  double bnum = 0.0;
  long long bden = 1;
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    // towards the greatest extreme if it limits there, else towards the least
    const long long den0 = tol3 - dV3[n], den1 = tol3 + dV3[n];   // 3 (tol -+ dV)
    const int h0 = __double2hiint(num[n][0]), h1 = __double2hiint(num[n][1]);
    const int key0 = ratio_key(num[n][0], den0, unit), key1 = ratio_key(num[n][1], den1, unit);
    const bool pos0 = h0 >= 0x100000, pos1 = h1 >= 0x100000;      // else zero, negative or denormal
    const bool in1 = den1 > 0 && (!pos1 || key1 < kKeyOne), in0 = den0 > 0 && (!pos0 || key0 < kKeyOne);
    // an extreme beyond the element's own mean by more than the slope goes past the tolerance
    past = past || (den1 <= 0 && h1 < 0 && key1 >= kKeyOne - kKeyClose) ||
           (!in1 && den0 <= 0 && h0 < 0 && key0 >= kKeyOne - kKeyClose);
    close = close || (den1 > 0 && pos1 && abs(key1 - kKeyOne) <= kKeyClose) ||
            (!in1 && den0 > 0 && pos0 && abs(key0 - kKeyOne) <= kKeyClose);
    const double q = in1 ? num[n][1] : num[n][0];
    const long long d = in1 ? den1 : den0;
    const int key = in1 ? key1 : key0;
    const bool in = in1 || in0, pos = in1 ? pos1 : pos0;
    zero = zero || (in && !pos);
    if (in && pos) {
      close = close || (abs(key - best) <= kKeyClose && (q != bnum || d != bden));
      if (key < best) { best = key; bnum = q; bden = d; }
    }
  }
  if (close) {                     // keys too close to tell: once more, exactly
    zero = past = false;
    best = kNone;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      bool open = true;
#pragma unroll
      for (int m = 1; m >= 0; --m) {
        const double q = num[n][m];
        const long long d = m ? tol3 + dV3[n] : tol3 - dV3[n];
        const bool pos = __double2hiint(q) >= 0x100000;
        past = past || (open && d <= 0 && __double2hiint(q) < 0 && ratio_key(q, d, unit) >= kKeyOne - kKeyClose);
        if (!open || d <= 0 || (pos && !below_one(q, d, unit))) continue;
        open = false;
        zero = zero || !pos;
        if (pos && (best == kNone || ratio_less(q, d, bnum, bden))) { best = 0; bnum = q; bden = d; }
      }
    }
  }
  if (past) return -1;
  if (zero) { alpha = 0.0; return 1; }
  if (best == kNone) return 0;
  const unsigned long long third = __umul64hi((unsigned long long)bden, 0xAAAAAAAAAAAAAAABULL) >> 1;   // bden / 3
  alpha = bnum / to_double((long long)third, unit);
  return alpha < 1.0 ? 1 : 0;
}

// Coefficients in digits, every order with a scale of its own: a derivative of order o at the barycentre
// is a sum over orders o and up (and of the tables' rounding below them), which differ by a power of
// the mesh width each.
template <int P> struct Orders {
  static constexpr int N = Dims<P>::N;
  __host__ __device__ static constexpr int begin(int s) { return s * (s + 1) / 2; }
  Dig d[N];
  int E[P + 1];
  __device__ __forceinline__ bool load(const double *c) {   // false: left to FP64
    bool ok = scale_of<1>(c, E[0]);
    if constexpr (P >= 1) ok = scale_of<2>(c + 1, E[1]) && ok;
    if constexpr (P >= 2) ok = scale_of<3>(c + 3, E[2]) && ok;
    if constexpr (P >= 3) ok = scale_of<4>(c + 6, E[3]) && ok;
#pragma unroll
    for (int s = 0; s <= P; ++s)
#pragma unroll
      for (int j = begin(s); j < begin(s + 1); ++j) d[j] = digits_of(c[j], max(E[s], kExpLo));
    return ok;
  }
  // u_i = sum_j DM_ij c_j for i in [I0, I1)
  template <int I0, int I1> __device__ __forceinline__ void derivatives(const FxTab<P> &tb, double *u) const {
#pragma unroll
    for (int i = I0; i < I1; ++i) {
      long long part[P + 1], v = 0;
      int x[P + 1], top = 0;
#pragma unroll
      for (int s = 0; s <= P; ++s) {
        Sum t;
#pragma unroll
        for (int j = begin(s); j < begin(s + 1); ++j) t.add(tb.DM[i][j], d[j]);
        part[s] = t.template over<29>();           // below 2^60, unit 2^(x - 1022 - 60)
        x[s] = E[s] ? E[s] + tb.eDM[i][s] : 0;
        top = max(top, x[s]);
      }
#pragma unroll
      for (int s = 0; s <= P; ++s) v += shr(part[s], top - x[s]);
      u[i] = to_double_int(v, top - 1022 - 60);
    }
  }
};

// Solution limiting of c in place (limit_lin_tile): where limited, the linear Taylor polynomial
// (u0, alpha u_1, alpha u_2) in the modal basis, u0 being the element's mean.  False: left to FP64, c
// untouched.
template <int P>
__device__ __forceinline__ bool linear_limit(const FxTab<P> &tb, const double lo[3], const double hi[3], int dmask,
                                             const double data[3], double u0, double *c) {
  constexpr int N = Dims<P>::N;
  Orders<P> o;
  if (!o.load(c)) return false;
  double u[3] = {u0, 0.0, 0.0}, alpha;
  o.template derivatives<1, 3>(tb, u);
  const int how = linear_alpha(lo, hi, dmask, data, u, alpha);
  if (how <= 0) return how == 0;
  u[1] *= alpha;
  u[2] *= alpha;
  int E0, E1;
  if (!scale_of<1>(u, E0) || !scale_of<2>(u + 1, E1)) return false;
  const Dig d0 = digits_of(u[0], max(E0, kExpLo)), d1 = digits_of(u[1], max(E1, kExpLo)), d2 = digits_of(u[2], max(E1, kExpLo));
#pragma unroll
  for (int i = 0; i < N; ++i) {
    Sum a, b;
    a.add(tb.DMi[i][0], d0);
    b.add(tb.DMi[i][1], d1);
    b.add(tb.DMi[i][2], d2);
    const int xa = E0 ? E0 + tb.eDMi[i][0] : 0, xb = E1 ? E1 + tb.eDMi[i][1] : 0, x = max(xa, xb);
    c[i] = to_double_int(shr(a.over<28>(), x - xa) + shr(b.over<28>(), x - xb), x - 1022 - 61);
  }
  return true;
}

// The exponents of an element's correction rows Q_k: word 0 the largest (negative: not in fixed
// point), then N bytes below it for the columns of each order of derivatives.
template <int P> struct CorrExp {
  static constexpr int N = Dims<P>::N, kWords = corr_exp_words(P) - 1;
  int head = -1;
  unsigned w[kWords];
  __device__ __forceinline__ void load(const int *__restrict__ qx, int Kp, int k) {
    head = qx[k];
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = (unsigned)qx[(size_t)(1 + i) * Kp + k];
  }
  __device__ __forceinline__ int at(int i) const { return head - byte_of(w, i); }
};
// Time-derivative limiting of cd (N coefficients, in place): cd += Q_k du (limit_dot_lin_tile), du the
// part of the reference derivatives that the limiter takes off, u0 the mean.
// sQ: digits of Q_k, row i (N-1) + (j-1), stride st.  False: left to FP64, cd untouched.
template <int P>
__device__ __forceinline__ bool linear_cdot_limit(const FxTab<P> &tb, const double lo[3], const double hi[3],
                                                  const Dig *sQ, int st, const CorrExp<P> &qx, double u0, double *cd) {
  constexpr int N = Dims<P>::N;
  if (qx.head < 0) return false;
  Orders<P> o;
  if (!o.load(cd)) return false;
  double w[N] = {u0}, alpha;
  o.template derivatives<1, 3>(tb, w);
  const double none[3] = {0.0, 0.0, 0.0};
  const int how = linear_alpha(lo, hi, 0, none, w, alpha);
  if (how <= 0) return how == 0;
  o.template derivatives<3, N>(tb, w);
  w[1] = (1.0 - alpha) * w[1];
  w[2] = (1.0 - alpha) * w[2];
  Dig du[N];
  int E[P];
  bool ok = scale_of<2>(w + 1, E[0]);
  if constexpr (P >= 2) ok = scale_of<3>(w + 3, E[1]) && ok;
  if constexpr (P >= 3) ok = scale_of<4>(w + 6, E[2]) && ok;
#pragma unroll
  for (int s = 0; s < P; ++s)
#pragma unroll
    for (int j = Orders<P>::begin(s + 1); j < Orders<P>::begin(s + 2); ++j) du[j] = digits_of(w[j], max(E[s], kExpLo));
  if (!ok) return false;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    long long part[P], v = 0;
    int xs[P], x = 0;
#pragma unroll
    for (int s = 0; s < P; ++s) {
      Sum t;
#pragma unroll
      for (int j = Orders<P>::begin(s + 1); j < Orders<P>::begin(s + 2); ++j) t.add(sQ[(size_t)(i * (N - 1) + (j - 1)) * st], du[j]);
      part[s] = t.template over<28>();
      xs[s] = E[s] ? E[s] + qx.at(s * N + i) : 0;
      x = max(x, xs[s]);
    }
#pragma unroll
    for (int s = 0; s < P; ++s) v += shr(part[s], x - xs[s]);
    cd[i] += to_double_int(v, x - 2044 - 61);
  }
  return true;
}
}  // namespace fx

// ---------------------------------------------------------------------------------------------
// The exponent below which a sum of magnitudes s lies (0: zero), and a byte below the base.
__device__ __forceinline__ int row_expo(double s, bool &ok) {
  const int e = fx::expo(s);
  if (s == 0.0) return 0;
  ok = ok && e >= fx::kMatLo && e <= fx::kExpHi;
  return e;
}
__device__ __forceinline__ int below(int e, int base, bool &ok) {
  if (e == 0) return 255;                          // a zero row or edge: any unit does
  ok = ok && base - e <= 255;
  return base - e;
}

// Digits of the element operator and the edge velocities of every element, their exponents and
// the element's inflow edges (OpExp).
template <int P>
__global__ void __launch_bounds__(128) k_fix_operator(int K, int Kp, const double *__restrict__ A,
                                                      const double *__restrict__ Vn, const int *__restrict__ nbr,
                                                      Dig *__restrict__ Ax, Dig *__restrict__ Vx, int *__restrict__ ax) {
  constexpr int N = Dims<P>::N, R = Dims<P>::R;
  using X = fx::OpExp<P>;
  const int k = blockIdx.x * 128 + threadIdx.x;
  if (k >= K) return;
  int e[4 * X::kWords] = {}, base = 0, in = 0;
  bool ok = true;
  for (int i = 0; i < N; ++i)
    for (int s = 0; s < X::kParts; ++s) {
      double sum = 0.0;
      for (int j = X::begin(s); j < X::begin(s + 1); ++j) sum += fabs(A[(size_t)(i * N + j) * Kp + k]);
      e[s * N + i] = row_expo(sum, ok);
      base = max(base, e[s * N + i]);
    }
  for (int n = 0; n < 3; ++n) {
    double vmax = 0.0;
    for (int r = 0; r < R; ++r) {
      const double v = Vn[(size_t)(n * R + r) * Kp + k];
      ok = ok && fx::finite_bits(v);
      vmax = fmax(vmax, fabs(v));
      if (v < 0.0 && nbr[(size_t)n * Kp + k] >= 0) in |= 1 << n;
    }
    e[X::kEdge + n] = row_expo(vmax, ok);
    base = max(base, e[X::kEdge + n]);
  }
  for (int i = 0; i < X::kWords; ++i) {
    unsigned w = 0;
    for (int b = 0; b < 4; ++b)
      if (4 * i + b < X::kEdge + 3) w |= (unsigned)(below(e[4 * i + b], base, ok) & 255) << (8 * b);
    ax[(size_t)(1 + i) * Kp + k] = (int)w;
  }
  ax[k] = (int)((ok ? 0u : 0x80000000u) | (unsigned)(in << 22) | (unsigned)base);
  for (int i = 0; i < N; ++i)
    for (int s = 0; s < X::kParts; ++s)
      for (int j = X::begin(s); j < X::begin(s + 1); ++j) {
        const size_t at = (size_t)(i * N + j) * Kp + k;
        const int E = e[s * N + i];
        Ax[at] = ok && E ? fx::digits_near(A[at], E) : Dig{0, 0};
      }
  for (int i = 0; i < 3 * R; ++i) {
    const size_t at = (size_t)i * Kp + k;
    const int E = e[X::kEdge + i / R];
    Vx[at] = ok && E ? fx::digits_near(Vn[at], E) : Dig{0, 0};
  }
}

// Digits of the correction rows Q_k and their exponents (CorrExp).
template <int P>
__global__ void __launch_bounds__(128) k_fix_correction(int K, int Kp, const double *__restrict__ Q,
                                                        Dig *__restrict__ Qx, int *__restrict__ qx) {
  constexpr int N = Dims<P>::N;
  using X = fx::CorrExp<P>;
  const int k = blockIdx.x * 128 + threadIdx.x;
  if (k >= K) return;
  int e[4 * X::kWords] = {}, base = 0;
  bool ok = true;
  for (int i = 0; i < N; ++i)
    for (int s = 0; s < P; ++s) {
      double sum = 0.0;
      for (int j = fx::Orders<P>::begin(s + 1); j < fx::Orders<P>::begin(s + 2); ++j) sum += fabs(Q[(size_t)(i * (N - 1) + j - 1) * Kp + k]);
      e[s * N + i] = row_expo(sum, ok);
      base = max(base, e[s * N + i]);
    }
  for (int i = 0; i < X::kWords; ++i) {
    unsigned w = 0;
    for (int b = 0; b < 4; ++b)
      if (4 * i + b < P * N) w |= (unsigned)(below(e[4 * i + b], base, ok) & 255) << (8 * b);
    qx[(size_t)(1 + i) * Kp + k] = (int)w;
  }
  qx[k] = ok ? base : -1;
  for (int i = 0; i < N; ++i)
    for (int j = 1; j < N; ++j) {
      const size_t at = (size_t)(i * (N - 1) + j - 1) * Kp + k;
      const int E = e[(j < 3 ? 0 : j < 6 ? N : 2 * N) + i];
      Qx[at] = ok && E ? fx::digits_near(Q[at], E) : Dig{0, 0};
    }
}

// ---------------------------------------------------------------------------------------------
// The digit tables (FxTab) from the FP64 tables, on the host.
inline int host_exponent(double x) {   // the least E with x <= 2^E
  int e = 0;
  if (x > 0.0 && std::frexp(x, &e) == 0.5) --e;
  return e;
}
template <int P>
inline void fill_digit_tables(const Tab<double, P> &t, FxTab<P> &f) {
  constexpr int N = Dims<P>::N, R = Dims<P>::R;
  double rowT = 0.0;
  for (int n = 0; n < 3; ++n)
    for (int np = 0; np < 3; ++np)
      for (int r = 0; r < R; ++r) {
        double s = 0.0;
        for (int j = 0; j < N; ++j) s += std::fabs(t.thetaPhi[n][np][r][j]);
        rowT = std::max(rowT, s);
      }
  f.eT = host_exponent(rowT);
  for (int i = 0; i < N; ++i) {
    for (int n = 0; n < 3; ++n) {
      double s = 0.0;
      for (int r = 0; r < R; ++r) s += std::fabs(t.Fphi[n][r][i]);
      f.eF[n][i] = host_exponent(s);
    }
    for (int n = 0; n < 3; ++n)
      for (int r = 0; r < R; ++r) {
        f.Fphi[n][r][i] = fx::digits_near(t.Fphi[n][r][i], f.eF[n][i] + 1022);
        for (int np = 0; np < 3; ++np) f.thetaPhi[n][np][r][i] = fx::digits_near(t.thetaPhi[n][np][r][i], f.eT + 1022);
      }
    for (int o = 0; o <= P; ++o) {
      const int b = fx::Orders<P>::begin(o), e = fx::Orders<P>::begin(o + 1);
      double a = 0.0;
      for (int j = b; j < e; ++j) a += std::fabs(t.DM[i][j]);
      f.eDM[i][o] = host_exponent(a);
      for (int j = b; j < e; ++j) f.DM[i][j] = fx::digits_near(t.DM[i][j], f.eDM[i][o] + 1022);
    }
    for (int o = 0; o < 2 && o <= P; ++o) {
      const int b = fx::Orders<P>::begin(o), e = fx::Orders<P>::begin(o + 1);
      double a = 0.0;
      for (int j = b; j < e; ++j) a += std::fabs(t.DMinv[i][j]);
      f.eDMi[i][o] = host_exponent(a);
      for (int j = b; j < e; ++j) f.DMi[i][j] = fx::digits_near(t.DMinv[i][j], f.eDMi[i][o] + 1022);
    }
  }
}

}  // namespace dgadv
