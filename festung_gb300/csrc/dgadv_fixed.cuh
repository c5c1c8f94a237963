// FP64 sums of products on the integer units.
//
// GB300 issues one FP64 instruction (multiply-add, add, compare, minimum alike) per 19 cycles
// and SM, but a 32 x 32 + 64 bit integer multiply-add every half cycle (both measured, all warps
// resident).  The FP64 stage kernels were bound by their sums of products with per-element or
// constant matrices, so those run in fixed point: the factors of a sum are scaled by common powers
// of two to 57-bit integers, each kept as two signed digits x = h 2^29 + l, |l| < 2^29.  A product
// is three of its four digit products (the low one is at most 2^-56 of the scale), accumulated
// without rounding in two 64-bit words: about 1.5 cycles instead of 19.  Everything that is not a
// sum of products (the Runge-Kutta update, the limiter's division) stays in FP64, whose pipe runs
// beside the integer units.
//
// Error.  With |a_j| scaled by their sum (a row of the matrix) and |x_j| by their maximum, a sum
// is off by at most about 2^-57 (sum |a_j|) max |x_j|, against 2^-53 sum |a_j x_j| and more for
// the FP64 chain.  Scales are per element, so values of very different size in different places
// keep their relative accuracy; an element whose exponents lie outside 2^(+-400), or that holds
// an infinity or a NaN, is left to the FP64 form of the same terms.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "dgadv_kernels.cuh"

namespace dgadv {

// The constant tables of a degree in digits: defined by the FP64 unit.
template <int P> __device__ __forceinline__ const FxTab<P> &fx_tab();

namespace fx {

constexpr int kW = 57;                       // bits of a scaled factor
constexpr int kExpLo = 623, kExpHi = 1423;   // biased exponents taken: 2^-400 .. 2^400

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
__device__ __forceinline__ Dig digits(long long X) {
  Dig d;
  d.l = (int)((unsigned)X << 3) >> 3;
  d.h = (int)((X - d.l) >> 29);
  return d;
}
// The digits of x in units of 2^(E - 1022 - kW): both of the sign of x, |l| < 2^29.
__device__ __forceinline__ Dig digits_of(double x, int E) {
  const unsigned long long v = fix_mag<kW>(x, E);
  const int sg = __double2hiint(x) >> 31;
  Dig d;
  d.l = ((int)((unsigned)v & 0x1fffffffu) ^ sg) - sg;
  d.h = ((int)(v >> 29) ^ sg) - sg;
  return d;
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
// The largest exponent among n values.
template <int n> __device__ __forceinline__ int max_expo(const double *x) {
  int e = 0;
#pragma unroll
  for (int j = 0; j < n; ++j) e = max(e, __double2hiint(x[j]) & 0x7fffffff);
  return e >> 20;
}

// Running sum: h 2^58 + m 2^29 in units of the factors' product.
struct Sum {
  long long h = 0, m = 0;
  __device__ __forceinline__ void add(const Dig &a, const Dig &b) {
    h += (long long)a.h * b.h;
    m += (long long)a.h * b.l;
    m += (long long)a.l * b.h;
  }
  // the sum over 2^(29 + S)
  template <int S> __device__ __forceinline__ long long over() const {
    static_assert(S >= 0 && S <= 29, "");
    return (h << (29 - S)) + (m >> S);
  }
};
__device__ __forceinline__ long long shr(long long x, int s) {   // x >> s for s of either sign
  return s >= 0 ? x >> min(s, 63) : x << min(-s, 63);
}

// ---------------------------------------------------------------------------------------------
// cDot of one element from its element operator: A c - sum over the inflow edges' points of
// Fphi v trace(neighbour) (stage_op_tile, kOpElement).
//   sA, sV: digits of A (row i N + j) and of v (row n R + r), row stride st
//   ax: exponents of A (bits 0..10, of its largest row sum) and v (11..21), inflow edges (22..24),
//       bit 31: not in fixed point
// Returns false (cdot untouched) where the element is left to FP64.
template <int P>
__device__ __forceinline__ bool element_cdot(const FxTab<P> &tb, const Dig *sA, const Dig *sV, int st, int ax,
                                             const double *c, const double (*cn)[Dims<P>::N], int code,
                                             double *cdot) {
  constexpr int N = Dims<P>::N, R = Dims<P>::R;
  if (ax < 0) return false;
  int E = max_expo<N>(c);
#pragma unroll
  for (int n = 0; n < 3; ++n)
    if ((ax >> (22 + n)) & 1) E = max(E, max_expo<N>(cn[n]));
  if (E == 0) {          // zero all over (a denormal goes to FP64)
    long long any = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      any |= __double_as_longlong(c[j]) << 1;
#pragma unroll
      for (int n = 0; n < 3; ++n)
        if ((ax >> (22 + n)) & 1) any |= __double_as_longlong(cn[n][j]) << 1;
    }
    if (any) return false;
#pragma unroll
    for (int i = 0; i < N; ++i) cdot[i] = 0.0;
    return true;
  }
  if (E < kExpLo || E > kExpHi) return false;
  const int Ea = ax & 2047, Ev = (ax >> 11) & 2047;
  long long acc[N];
  {
    Dig d[N];
#pragma unroll
    for (int j = 0; j < N; ++j) d[j] = digits_of(c[j], E);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Sum s;
#pragma unroll
      for (int j = 0; j < N; ++j) s.add(sA[(size_t)(i * N + j) * st], d[j]);
      acc[i] = s.over<24>();                       // below 2^61, unit 2^(ea + ec - 61)
    }
  }
  int unit = (Ea - 1022) + (E - 1022) - 61;
  if ((ax >> 22) & 7) {
    Sum f[N];
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      if (!((ax >> (22 + n)) & 1)) continue;
      const int np = (code >> (2 * n)) & 3;
      Dig d[N];
#pragma unroll
      for (int j = 0; j < N; ++j) d[j] = digits_of(cn[n][j], E);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const Dig v = sV[(size_t)(n * R + r) * st];
        if (!(v.h < 0 || (v.h == 0 && v.l < 0))) continue;
        Sum tr, fl;
#pragma unroll
        for (int j = 0; j < N; ++j) tr.add(tb.thetaPhi[n][np][r][j], d[j]);
        fl.add(digits(tr.over<26>()), v);          // trace below 2^59, unit 2^(ec + eT - 59)
        const Dig q = digits(-fl.over<28>());      // below 2^59, unit 2^(ec + eT + ev - 59)
#pragma unroll
        for (int i = 0; i < N; ++i) f[i].add(tb.Fphi[n][r][i], q);
      }
    }
    // unit 2^(ec + eT + ev + eF - 61): both parts in the coarser unit of the two
    const int D = tb.eT + tb.eF + Ev - Ea;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const long long w = f[i].template over<26>();
      acc[i] = D > 0 ? (acc[i] >> min(D, 63)) + w : acc[i] + (w >> min(-D, 63));
    }
    unit += max(D, 0);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) cdot[i] = to_double(acc[i], unit);
  return true;
}

// ---------------------------------------------------------------------------------------------
// The linear limiter's factor (vertex_alpha_1div) for u_0, u_1, u_2 given as u[i] 2^(uu[i]) and the
// patch extremes (shifted), in integers of one unit, 2^(G - 1082), that holds them all: the
// differences, comparisons and cross products are exact.  G is the largest exponent among the
// extremes and u, so the unit is 2^-60 of the largest value, where FP64 rounds at 2^-53 of each.
// Returns 0: not limited, 1: limited by alpha, -1: left to FP64.
__device__ __forceinline__ int linear_alpha(const double lo[3], const double hi[3], int dmask, const double data[3],
                                            const long long u[3], const int uu[3], double &alpha) {
  int S = 1000;                                   // the tolerance 1e-8 (exponent 996) fits the unit
#pragma unroll
  for (int n = 0; n < 3; ++n) S = max(S, max(expo(lo[n]), expo(hi[n])));
  if (S > kExpHi) return -1;
  int G = S;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const long long m = u[i] < 0 ? ~u[i] : u[i];
    G = max(G, 64 - __clzll(m) + uu[i] + 1022);   // |u_i| < 2^(G - 1022)
  }
  long long dat[3] = {0, 0, 0};
  if (dmask) {
#pragma unroll
    for (int n = 0; n < 3; ++n)
      if ((dmask >> n) & 1) {
        G = max(G, expo(data[n]));
      }
  }
  if (G > S + 6) return -1;                       // slopes far above the means: the unit would be too coarse
  const int g = G - 1022 - 60;
  long long U[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) U[i] = shr(u[i], g - uu[i]);
  if (dmask) {
#pragma unroll
    for (int n = 0; n < 3; ++n) dat[n] = fix<60>(data[n], G);
  }
  const long long tol3 = 3 * fix<60>(1.e-8, G);
  const long long dV3[3] = {-(U[1] + U[2]), 2 * U[1] - U[2], 2 * U[2] - U[1]};
  unsigned long long bn = 0, bd = 1;
  bool any = false;
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    long long mn = fix<60>(lo[n], G), mx = fix<60>(hi[n], G);
    if ((dmask >> n) & 1) { mn = min(mn, dat[n]); mx = max(mx, dat[n]); }
    const long long dMin3 = 3 * (mn - U[0]), dMax3 = 3 * (mx - U[0]);
    long long num = 0, den = 1;
    bool br = false;
    if (dV3[n] < dMin3 + tol3) { num = -dMin3; den = tol3 - dV3[n]; br = true; }
    if (dV3[n] > dMax3 - tol3) { num = dMax3; den = dV3[n] + tol3; br = true; }
    if (br) {
      if (den <= 0) return -1;                    // an extreme rounded past the element's own value
      const unsigned long long un = num > 0 ? (unsigned long long)num : 0ULL, ud = (unsigned long long)den;
      if (!any || (unsigned __int128)un * bd < (unsigned __int128)bn * ud) { bn = un; bd = ud; any = true; }
    }
  }
  if (!any || bn >= bd) return 0;
  alpha = to_double((long long)bn) / to_double((long long)bd);
  return alpha == 1.0 ? 0 : 1;
}


// The sums of linear_cdot_limit and linear_limit below: u_j = sum_k DM_jk x_k for j in [J0, J1), as
// u[j] 2^(E - 1022 + eDM_j - 58).
template <int P, int J0, int J1>
__device__ __forceinline__ void reference_derivatives(const FxTab<P> &tb, const Dig *d, long long *u) {
  constexpr int N = Dims<P>::N;
#pragma unroll
  for (int i = J0; i < (J1 < N ? J1 : N); ++i) {
    Sum s;
#pragma unroll
    for (int j = 0; j < N; ++j) s.add(tb.DM[i][j], d[j]);
    u[i] = s.over<27>();
  }
}

// Time-derivative limiting of cd (N coefficients, in place): cd += Q_k du (limit_dot_lin_tile).
// sQ: digits of Q_k with column j scaled by 2^(eDM_j), row i (N-1) + (j-1), stride st; qx: the
// exponent of its largest row sum (negative: not in fixed point).  False: left to FP64.
template <int P>
__device__ __forceinline__ bool linear_cdot_limit(const FxTab<P> &tb, const double lo[3], const double hi[3],
                                                  const Dig *sQ, int st, int qx, double *cd) {
  constexpr int N = Dims<P>::N;
  int E = max_expo<N>(cd);
  if (qx < 0 || E > kExpHi) return false;
  E = max(E, kExpLo);                              // what is below 2^-457 counts as zero
  Dig d[N];
#pragma unroll
  for (int j = 0; j < N; ++j) d[j] = digits_of(cd[j], E);
  long long u[N];
  reference_derivatives<P, 0, 3>(tb, d, u);
  const int uu[3] = {E - 1022 + tb.eDM[0] - 58, E - 1022 + tb.eDM[1] - 58, E - 1022 + tb.eDM[2] - 58};
  double alpha;
  const double none[3] = {0.0, 0.0, 0.0};
  const int how = linear_alpha(lo, hi, 0, none, u, uu, alpha);
  if (how <= 0) return how == 0;
  reference_derivatives<P, 3, N>(tb, d, u);
  const Dig om = digits_of(1.0 - alpha, 1023);   // (1 - alpha) 2^56
  Dig du[N];
#pragma unroll
  for (int j = 1; j < N; ++j) {
    if (j < 3) {
      Sum s;
      s.add(digits(u[j]), om);
      u[j] = s.over<27>();
    }
    du[j] = digits(u[j]);
  }
  const int q = qx - 1022;                          // Q du in units 2^(q + ec - 61), cd in 2^(ec - 57)
  const int sh = max(q, 0);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    Sum s;
#pragma unroll
    for (int j = 1; j < N; ++j) s.add(sQ[(size_t)(i * (N - 1) + (j - 1)) * st], du[j]);
    const long long c = (long long)d[i].h * (1LL << 29) + d[i].l;
    cd[i] = to_double_int(shr(c, sh - 4) + shr(s.over<25>(), sh - q), E - 1022 - 61 + sh);
  }
  return true;
}

// Solution limiting of c in place (limit_lin_tile): where limited, the linear Taylor polynomial
// (u_0, alpha u_1, alpha u_2) in the modal basis.  False: left to FP64.
template <int P>
__device__ __forceinline__ bool linear_limit(const FxTab<P> &tb, const double lo[3], const double hi[3], int dmask,
                                             const double data[3], double *c) {
  constexpr int N = Dims<P>::N;
  int E = max_expo<N>(c);
  if (E > kExpHi) return false;
  E = max(E, kExpLo);
  Dig d[N];
#pragma unroll
  for (int j = 0; j < N; ++j) d[j] = digits_of(c[j], E);
  long long u[3];
  reference_derivatives<P, 0, 3>(tb, d, u);
  const int uu[3] = {E - 1022 + tb.eDM[0] - 58, E - 1022 + tb.eDM[1] - 58, E - 1022 + tb.eDM[2] - 58};
  double alpha;
  const int how = linear_alpha(lo, hi, dmask, data, u, uu, alpha);
  if (how <= 0) return how == 0;
  const Dig al = digits_of(alpha, 1023);
  Dig w[3] = {digits(u[0]), {0, 0}, {0, 0}};
#pragma unroll
  for (int j = 1; j < 3; ++j) {
    Sum s;
    s.add(digits(u[j]), al);
    w[j] = digits(s.over<27>());
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    Sum s;
#pragma unroll
    for (int j = 0; j < 3; ++j) s.add(tb.DMi[i][j], w[j]);
    c[i] = to_double(s.over<25>(), E - 1022 + tb.eDMi[i] - 61);
  }
  return true;
}
}  // namespace fx

// Digits of the element operator and the edge velocities of every element, their exponents and
// the element's inflow edges (element_cdot's ax).
template <int P>
__global__ void __launch_bounds__(128) k_fix_operator(int K, int Kp, const double *__restrict__ A,
                                                      const double *__restrict__ Vn, const int *__restrict__ nbr,
                                                      Dig *__restrict__ Ax, Dig *__restrict__ Vx, int *__restrict__ ax) {
  constexpr int N = Dims<P>::N, R = Dims<P>::R;
  const int k = blockIdx.x * 128 + threadIdx.x;
  if (k >= K) return;
  double big = 0.0, vmax = 0.0;
  bool ok = true;
  for (int i = 0; i < N; ++i) {
    double s = 0.0;
    for (int j = 0; j < N; ++j) s += fabs(A[(size_t)(i * N + j) * Kp + k]);
    ok = ok && fx::finite_bits(s);
    big = fmax(big, s);
  }
  int in = 0;
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < R; ++r) {
      const double v = Vn[(size_t)(n * R + r) * Kp + k];
      ok = ok && fx::finite_bits(v);
      vmax = fmax(vmax, fabs(v));
      if (v < 0.0 && nbr[(size_t)n * Kp + k] >= 0) in |= 1 << n;
    }
  const int Ea = big == 0.0 ? 1023 : fx::expo(big), Ev = vmax == 0.0 ? 1023 : fx::expo(vmax);
  ok = ok && Ea >= fx::kExpLo && Ea <= fx::kExpHi && Ev >= fx::kExpLo && Ev <= fx::kExpHi;
  ax[k] = ok ? (Ea | (Ev << 11) | (in << 22)) : (int)(0x80000000u | (unsigned)(in << 22));
  for (int i = 0; i < N * N; ++i) Ax[(size_t)i * Kp + k] = fx::digits(ok ? fx::fix<fx::kW>(A[(size_t)i * Kp + k], Ea) : 0);
  for (int i = 0; i < 3 * R; ++i) Vx[(size_t)i * Kp + k] = fx::digits(ok ? fx::fix<fx::kW>(Vn[(size_t)i * Kp + k], Ev) : 0);
}

// Digits of the correction rows Q_k, column j scaled by 2^(eDM_j), and the exponent of the
// element's largest row sum (-1: not in fixed point).
template <int P>
__global__ void __launch_bounds__(128) k_fix_correction(int K, int Kp, const double *__restrict__ Q,
                                                        Dig *__restrict__ Qx, int *__restrict__ qx) {
  constexpr int N = Dims<P>::N;
  const FxTab<P> &tb = fx_tab<P>();
  const int k = blockIdx.x * 128 + threadIdx.x;
  if (k >= K) return;
  double big = 0.0;
  for (int i = 0; i < N; ++i) {
    double s = 0.0;
    for (int j = 1; j < N; ++j) s += fabs(ldexp(Q[(size_t)(i * (N - 1) + j - 1) * Kp + k], tb.eDM[j]));
    big = fx::finite_bits(s) ? fmax(big, s) : INFINITY;
  }
  const int E = big == 0.0 ? 1023 : fx::expo(big);
  const bool ok = E >= fx::kExpLo && E <= fx::kExpHi;
  qx[k] = ok ? E : -1;
  for (int i = 0; i < N; ++i)
    for (int j = 1; j < N; ++j) {
      const size_t at = (size_t)(i * (N - 1) + j - 1) * Kp + k;
      Qx[at] = fx::digits(ok ? fx::fix<fx::kW>(ldexp(Q[at], tb.eDM[j]), E) : 0);
    }
}

}  // namespace dgadv
