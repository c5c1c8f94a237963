// The FP64 kernels' fixed-point arithmetic (festung_gb300/csrc/dgadv_fixed.cuh) on the host: the header
// compiled as it is, with the few device intrinsics it uses written out below.  Every entry point
// evaluates one element operation three ways, in fixed point, as the kernels' FP64 multiply-add chain and
// in long double (64-bit mantissa on x86-64), and returns both errors beside the sum of the terms'
// magnitudes.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __forceinline__
#define __forceinline__ inline

static struct { int x = 0, y = 0; } blockIdx, threadIdx;
static long long __double_as_longlong(double x) { long long r; std::memcpy(&r, &x, 8); return r; }
static double __longlong_as_double(long long x) { double r; std::memcpy(&r, &x, 8); return r; }
static int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
static int __double2loint(double x) { return (int)__double_as_longlong(x); }
static double __hiloint2double(int h, int l) {
  return __longlong_as_double((long long)(((unsigned long long)(unsigned)h << 32) | (unsigned)l));
}
static int __clzll(long long x) { return x == 0 ? 64 : __builtin_clzll((unsigned long long)x); }
static unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
static float __int_as_float(int x) { float r; std::memcpy(&r, &x, 4); return r; }
static int __float_as_int(float x) { int r; std::memcpy(&r, &x, 4); return r; }
static float __fdividef(float a, float b) { return a / b; }
static float __ll2float_rn(long long x) { return (float)x; }
using std::max;
using std::min;

#include "dgadv_fixed.cuh"
#include "dgadv_tables.h"

namespace dgadv {
template <int P> FxTab<P> &host_fx() { static FxTab<P> t; return t; }
template <> const FxTab<0> &fx_tab<0>() { return host_fx<0>(); }
template <> const FxTab<1> &fx_tab<1>() { return host_fx<1>(); }
template <> const FxTab<2> &fx_tab<2>() { return host_fx<2>(); }
template <> const FxTab<3> &fx_tab<3>() { return host_fx<3>(); }
}  // namespace dgadv
using namespace dgadv;

namespace {
typedef long double Wide;

struct Out {
  double *value, *errFixed, *errFp64, *size;   // K x N each
  int32_t *taken;                              // K: done in fixed point
  void set(int i, double v, double fp64, Wide exact, Wide s) const {
    value[i] = v;
    errFixed[i] = (double)std::fabs(v - exact);
    errFp64[i] = (double)std::fabs(fp64 - exact);
    size[i] = (double)s;
  }
};

// cDot of every element; velocity 0: rotation about the centre, 1: exp((x + y) / 2), exp((x - y) / 2);
// edge n of element k scaled by vScale[3 k + n] (the element's own side).
template <int P>
int run_operator(const Grid &gr, int velocity, const double *vScale, const double *c, const Out &o) {
  constexpr int N = Dims<P>::N, Q = Dims<P>::Q, R = Dims<P>::R;
  RefTables rt;
  std::string err;
  if (!build_ref_tables(P, rt, err)) return 1;
  Tab<double, P> tb;
  fill_tables(rt, tb);
  fill_digit_tables(tb, host_fx<P>());
  for (int e = 0; e < gr.numT; ++e) {
    const double *X = &gr.coordV0T[6 * (size_t)e], *B = &gr.B[4 * (size_t)e], dj = gr.detJ0T[e];
    auto vel = [&](double s, double t, double &a, double &b) {
      const double x = X[0] + (X[2] - X[0]) * s + (X[4] - X[0]) * t, y = X[1] + (X[3] - X[1]) * s + (X[5] - X[1]) * t;
      a = velocity ? std::exp(0.5 * (x + y)) : 0.5 - y;
      b = velocity ? std::exp(0.5 * (x - y)) : x - 0.5;
    };
    double F[2][Q], v[3 * R], a, b;
    for (int q = 0; q < Q; ++q) {
      vel(rt.vol.Q1[q], rt.vol.Q2[q], a, b);
      F[0][q] = rt.vol.W[q] * (B[3] * a - B[1] * b) / dj;
      F[1][q] = rt.vol.W[q] * (B[0] * b - B[2] * a) / dj;
    }
    int nb[3], np[3], code = 7 << 6;
    for (int n = 0; n < 3; ++n) {
      const int ed = gr.E0T[3 * (size_t)e + n], side = gr.T0E[2 * (size_t)ed] == e ? 1 : 0;
      nb[n] = gr.T0E[2 * (size_t)ed + side];
      np[n] = std::max(0, gr.E0E[2 * (size_t)ed + side]);
      code |= np[n] << (2 * n);
      const double p0[2] = {n == 0 ? 1.0 : 0.0, n == 1 ? 1.0 : 0.0};   // edge n from corner n + 1 to n + 2
      const double p1[2] = {n == 2 ? 1.0 : 0.0, n == 0 ? 1.0 : 0.0};
      for (int r = 0; r < R; ++r) {
        const double t = rt.edge.Q[r];
        vel(p0[0] + (p1[0] - p0[0]) * t, p0[1] + (p1[1] - p0[1]) * t, a, b);
        v[n * R + r] = (vScale ? vScale[3 * (size_t)e + n] : 1.0) * gr.areaE0T[3 * (size_t)e + n] * rt.edge.W[r] *
                       (a * gr.nuE0T[6 * (size_t)e + 2 * n] + b * gr.nuE0T[6 * (size_t)e + 2 * n + 1]) / dj;
      }
    }
    double A[N * N];
    for (int i = 0; i < N; ++i)
      for (int j = 0; j < N; ++j) {
        double s = 0.0;
        for (int q = 0; q < Q; ++q) {
          s = std::fma(tb.Fg1[q][i] * F[0][q], tb.phiQ[q][j], s);
          s = std::fma(tb.Fg2[q][i] * F[1][q], tb.phiQ[q][j], s);
        }
        for (int x = 0; x < 3 * R; ++x)
          if (v[x] > 0.0) s = std::fma(-tb.Fphi[x / R][x % R][i] * v[x], tb.phi1D[x / R][x % R][j], s);
        A[i * N + j] = s;
      }
    const double *ce = c + (size_t)e * N;
    double cn[3][N] = {}, fp[N], fixed[N];
    Wide exact[N], size[N];
    for (int n = 0; n < 3; ++n)
      if (nb[n] >= 0) std::copy(c + (size_t)nb[n] * N, c + (size_t)(nb[n] + 1) * N, cn[n]);
    for (int i = 0; i < N; ++i) {
      fp[i] = 0.0; exact[i] = size[i] = 0;
      for (int j = 0; j < N; ++j) {
        fp[i] = std::fma(A[i * N + j], ce[j], fp[i]);
        exact[i] += (Wide)A[i * N + j] * ce[j];
        size[i] += std::fabs((Wide)A[i * N + j] * ce[j]);
      }
    }
    for (int x = 0; x < 3 * R; ++x) {
      const int n = x / R, r = x % R;
      if (!(v[x] < 0.0) || nb[n] < 0) continue;
      double tr = 0.0;
      Wide trw = 0, trs = 0;
      for (int j = 0; j < N; ++j) {
        tr = std::fma(tb.thetaPhi[n][np[n]][r][j], cn[n][j], tr);
        trw += (Wide)tb.thetaPhi[n][np[n]][r][j] * cn[n][j];
        trs += std::fabs((Wide)tb.thetaPhi[n][np[n]][r][j] * cn[n][j]);
      }
      const double fl = v[x] * tr;
      for (int i = 0; i < N; ++i) {
        fp[i] = std::fma(-tb.Fphi[n][r][i], fl, fp[i]);
        exact[i] -= (Wide)tb.Fphi[n][r][i] * v[x] * trw;
        size[i] += std::fabs((Wide)tb.Fphi[n][r][i] * v[x]) * trs;
      }
    }
    Dig ax[N * N], vx[3 * R];
    int words[op_exp_words(P)];
    k_fix_operator<P>(1, 1, A, v, nb, ax, vx, words);
    fx::OpExp<P> x;
    x.load(words, 1, 0);
    o.taken[e] = fx::element_cdot<P>(host_fx<P>(), ax, vx, 1, x, ce, cn, code, fixed);
    if (!o.taken[e]) std::copy(fp, fp + N, fixed);
    for (int i = 0; i < N; ++i) o.set(e * N + i, fixed[i], fp[i], exact[i], size[i]);
  }
  return 0;
}

template <typename T> T alpha_of(const double *lo, const double *hi, const T *u) {
  const T tol = 1e-8, third = T(1) / T(3), two3 = T(2) / T(3), hx[3] = {-third, two3, -third}, hy[3] = {-third, -third, two3};
  T a = 1;
  for (int n = 0; n < 3; ++n) {
    const T v = (u[0] + u[1] * hx[n]) + u[2] * hy[n], dV = v - u[0], dMin = lo[n] - u[0], dMax = hi[n] - u[0];
    T num = 1, den = 1;                        // towards the greatest extreme if both hold
    if (dV < dMin + tol) { num = -dMin; den = tol - dV; }
    if (dV > dMax - tol) { num = dMax; den = dV + tol; }
    a = std::min(a, std::max(T(0), num / den));
  }
  return a;
}

// The linear limiter of the time derivative, c <- c + Q du, and (solution) of the solution, c <- the
// linear polynomial, of every element from the extremes of its vertex patches.
template <int P>
int run_limiter(const Grid &gr, bool solution, const double *c, const Out &o) {
  constexpr int N = Dims<P>::N;
  RefTables rt;
  std::string err;
  if (!build_ref_tables(P, rt, err)) return 1;
  Tab<double, P> tb;
  fill_tables(rt, tb);
  fill_digit_tables(tb, host_fx<P>());
  std::vector<double> qk, vmin(gr.numV, INFINITY), vmax(gr.numV, -INFINITY);
  taylor_correction(gr, P, rt, qk);
  auto row = [&](const double *ce, int i) {
    double s = 0.0;
    for (int j = 0; j < N; ++j) s = std::fma(tb.DM[i][j], ce[j], s);
    return s;
  };
  for (int e = 0; e < gr.numT; ++e)
    for (int n = 0; n < 3; ++n) {
      const int w = gr.V0T[3 * (size_t)e + n];
      vmin[w] = std::min(vmin[w], row(c + (size_t)e * N, 0));
      vmax[w] = std::max(vmax[w], row(c + (size_t)e * N, 0));
    }
  for (int e = 0; e < gr.numT; ++e) {
    const double *ce = c + (size_t)e * N, *q = &qk[(size_t)e * N * (N - 1)];
    double lo[3], hi[3], u[N], fp[N], fixed[N];
    Wide U[N], exact[N], size[N];
    for (int n = 0; n < 3; ++n) { lo[n] = vmin[gr.V0T[3 * (size_t)e + n]]; hi[n] = vmax[gr.V0T[3 * (size_t)e + n]]; }
    for (int i = 0; i < N; ++i) {
      u[i] = row(ce, i);
      U[i] = 0;
      for (int j = 0; j < N; ++j) U[i] += (Wide)tb.DM[i][j] * ce[j];
      fp[i] = fixed[i] = ce[i];
      exact[i] = ce[i];
      size[i] = std::fabs(exact[i]);
    }
    const double a = alpha_of(lo, hi, u);
    const Wide UU[3] = {u[0], U[1], U[2]}, aw = alpha_of(lo, hi, UU);   // the mean as it was compared
    if (solution) {
      const double none[3] = {0.0, 0.0, 0.0};
      o.taken[e] = fx::linear_limit<P>(host_fx<P>(), lo, hi, 0, none, u[0], fixed);
      for (int i = 0; i < N; ++i) {
        if (a != 1.0) fp[i] = std::fma(tb.DMinv[i][2], a * u[2], std::fma(tb.DMinv[i][1], a * u[1], tb.DMinv[i][0] * u[0]));
        if (aw < 1) {
          exact[i] = tb.DMinv[i][0] * U[0] + aw * (tb.DMinv[i][1] * U[1] + tb.DMinv[i][2] * U[2]);
          size[i] = std::fabs(tb.DMinv[i][0] * U[0]) + std::fabs(aw * tb.DMinv[i][1] * U[1]) + std::fabs(aw * tb.DMinv[i][2] * U[2]);
        }
      }
      if (!o.taken[e]) std::copy(fp, fp + N, fixed);
    } else {
      Dig qd[N * (N - 1)];
      int words[corr_exp_words(P)];
      k_fix_correction<P>(1, 1, q, qd, words);
      fx::CorrExp<P> x;
      x.load(words, 1, 0);
      if (a != 1.0)
        for (int i = 0; i < N; ++i)
          for (int j = 1; j < N; ++j) fp[i] = std::fma(q[i * (N - 1) + j - 1], j < 3 ? (1.0 - a) * u[j] : u[j], fp[i]);
      if (aw < 1)
        for (int i = 0; i < N; ++i)
          for (int j = 1; j < N; ++j) {
            const Wide t = (Wide)q[i * (N - 1) + j - 1] * (j < 3 ? (1 - aw) * U[j] : U[j]);
            exact[i] += t;
            size[i] += std::fabs(t);
          }
      o.taken[e] = fx::linear_cdot_limit<P>(host_fx<P>(), lo, hi, qd, 1, x, u[0], fixed);
      if (!o.taken[e]) std::copy(fp, fp + N, fixed);
    }
    for (int i = 0; i < N; ++i) o.set(e * N + i, fixed[i], fp[i], exact[i], size[i]);
  }
  return 0;
}
}  // namespace

extern "C" int fixed_point_operator(int p, int numV, const double *coordV, int numT, const int32_t *V0T, int velocity,
                                    const double *vScale, const double *c, double *value, double *errFixed,
                                    double *errFp64, double *size, int32_t *taken) {
  Grid gr;
  std::string err;
  const Out o{value, errFixed, errFp64, size, taken};
  if (!build_grid(numV, coordV, numT, V0T, gr, err)) return 1;
  return p == 0 ? run_operator<0>(gr, velocity, vScale, c, o) : p == 1 ? run_operator<1>(gr, velocity, vScale, c, o)
       : p == 2 ? run_operator<2>(gr, velocity, vScale, c, o) : run_operator<3>(gr, velocity, vScale, c, o);
}

extern "C" int fixed_point_limiter(int p, int numV, const double *coordV, int numT, const int32_t *V0T, int solution,
                                   const double *c, double *value, double *errFixed, double *errFp64, double *size,
                                   int32_t *taken) {
  Grid gr;
  std::string err;
  const Out o{value, errFixed, errFp64, size, taken};
  if (!build_grid(numV, coordV, numT, V0T, gr, err)) return 1;
  return p == 2 ? run_limiter<2>(gr, solution != 0, c, o) : run_limiter<3>(gr, solution != 0, c, o);
}

// The sum of each 32 of x as the implicit solver's warps form it (57 bits below the largest exponent).
extern "C" void fixed_point_lane_sums(int n, const double *x, double *out) {
  for (int i = 0; i < n; ++i) {
    int E = 223;
    long long v = 0;
    for (int l = 0; l < 32; ++l) E = std::max(E, fx::expo(x[32 * i + l]));
    for (int l = 0; l < 32; ++l) v += fx::fix_near<57>(x[32 * i + l], E);
    out[i] = fx::to_double_int(v, E - 1022 - 57);
  }
}
