// The constant tables of a degree (Tab) from the reference tables, on the host.
#pragma once
#include "dgadv_host.h"
#include "dgadv_kernels.cuh"

namespace dgadv {

template <typename T, int P>
inline void fill_tables(const RefTables &rt, Tab<T, P> &t) {
  constexpr int N = Dims<P>::N, Q = Dims<P>::Q, R = Dims<P>::R;
  for (int q = 0; q < Q; ++q)
    for (int i = 0; i < N; ++i) {
      t.phiQ[q][i] = T(rt.phiQ[q * N + i]);
      t.g1[q][i] = T(rt.gradQ[q * N + i]);
      t.g2[q][i] = T(rt.gradQ[Q * N + q * N + i]);
    }
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < R; ++r)
      for (int i = 0; i < N; ++i) t.phi1D[n][r][i] = T(rt.phi1D[(n * R + r) * N + i]);
  for (int nn = 0; nn < 3; ++nn)
    for (int np = 0; np < 3; ++np)
      for (int r = 0; r < R; ++r)
        for (int i = 0; i < N; ++i) t.thetaPhi[nn][np][r][i] = T(rt.thetaPhi[((nn * 3 + np) * R + r) * N + i]);
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      t.hatMinv[i][j] = T(rt.hatMinv[i * N + j]);
      t.DM[i][j] = T(rt.DM[i * N + j]);
      t.DMinv[i][j] = T(rt.DMinv[i * N + j]);
    }
  // Gr = DM^-T hatM DM^-1 in FP64, then rounded
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      double s = 0.0;
      for (int a = 0; a < N; ++a) {
        double r = 0.0;
        for (int b = 0; b < N; ++b) r += rt.hatM[a * N + b] * rt.DMinv[b * N + j];
        s += rt.DMinv[a * N + i] * r;
      }
      t.Gr[i][j] = T(s);
    }
  // adjoint tables (the forward FP32 path takes hatM^-1 = I; so does its adjoint)
  const bool massSolve = sizeof(T) == 8;
  auto fold = [&](const double *row, int j) {
    if (!massSolve) return row[j];
    double a = 0.0;
    for (int i = 0; i < N; ++i) a += row[i] * rt.hatMinv[i * N + j];
    return a;
  };
  for (int q = 0; q < Q; ++q)
    for (int j = 0; j < N; ++j) {
      t.Hg1[q][j] = T(fold(&rt.gradQ[q * N], j));
      t.Hg2[q][j] = T(fold(&rt.gradQ[Q * N + q * N], j));
    }
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < R; ++r)
      for (int j = 0; j < N; ++j) t.Hphi[n][r][j] = T(fold(&rt.phi1D[(n * R + r) * N], j));
  // forward tables: hatM^-1 applied from the left, in FP64, then rounded
  auto lfold = [&](const double *row, int i) {
    if (!massSolve) return row[i];
    double a = 0.0;
    for (int j = 0; j < N; ++j) a += rt.hatMinv[i * N + j] * row[j];
    return a;
  };
  for (int q = 0; q < Q; ++q)
    for (int i = 0; i < N; ++i) {
      t.Fg1[q][i] = T(lfold(&rt.gradQ[q * N], i));
      t.Fg2[q][i] = T(lfold(&rt.gradQ[Q * N + q * N], i));
    }
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < R; ++r)
      for (int i = 0; i < N; ++i) t.Fphi[n][r][i] = T(lfold(&rt.phi1D[(n * R + r) * N], i));
}

}  // namespace dgadv
