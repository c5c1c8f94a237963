// Implicit time stepping: the advection_implicit problem on the device.
//
// The reference solves, per stage of a diagonally implicit Runge-Kutta method
// (core/rungeKuttaImplicit.m, advection_implicit/solveSubStep.m),
//     (M + tau a_ii A) x_i = tau a_ii sysV(t_i) + M c^n + sum_{j<i} tau a_ij rhs_j,
//     rhs_i = sysV(t_i) - A x_i,      c^{n+1} = x_S,
// and A x = sysV for a stationary problem, each with a sparse direct solver.  Here the same
// equations are multiplied by M^-1 (block diagonal) and solved matrix-free:
//     (I + tau a_ii M^-1 A) x_i = c^n + tau sum_{j<i} a_ij k_j + tau a_ii s_i,
//     s_i = M^-1 sysV(t_i),   k_i = s_i - M^-1 A x_i,
// by restarted GMRES with classical Gram-Schmidt twice, right-preconditioned by the inverse of
// each element's diagonal block.  The operator kernel is the stage operator's arithmetic
// (volume term, upwind flux, mass solve) with the implicit problem's volume rule of order 2p+1
// (advection_implicit/preprocessProblem.m); handles for it are created with
// DGADV_FLAG_IMPLICIT.  Vectors are the handle's SoA state layout (N x Kp, padding zero);
// inner products accumulate in FP64.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "dgadv_fixed.cuh"
#include "dgadv_handle.h"

namespace dgadv {
namespace {

constexpr int kImplBlock = 128;
// Every kernel over the elements runs blocks of 32 elements x N coefficient rows, a warp per row: FP64
// instructions issue at their full (low) rate only with warps on all four schedulers of an SM, and
// the reference's 8192 elements are 256 warps with a thread per element, under two per SM.  Larger meshes do
// not lose by it: 524288 elements, p = 1, 567 us per iteration with a thread per element, 397 so.
constexpr int kRows = 32;             // elements per block
constexpr int kVecs = 8;              // basis vectors a thread has in flight at once
constexpr int kCheck = 4;             // Arnoldi steps between two looks at the residual estimate
constexpr int kVecThreads = 256;
constexpr int kChunk = 8;             // vectors per linear combination launch

template <int P> struct IDims {
  static constexpr int N = (P + 1) * (P + 2) / 2;
  static constexpr int Q = P == 0 ? 1 : (P == 1 ? 4 : (P == 2 ? 7 : 49));   // quadRule2D(2p+1)
  static constexpr int R = P + 1;                                            // quadRule1D(2p+1)
};

template <typename T, int P> struct ImplTab {
  static constexpr int N = IDims<P>::N, Q = IDims<P>::Q, R = IDims<P>::R;
  T phiQ[Q][N];
  T g1[Q][N];
  T g2[Q][N];
  T phi1D[3][R][N];
  T thetaPhi[3][3][R][N];
  T hatMinv[N][N];
  T Fphi[3][R][N];    // hatM^-1 applied to the edge test functions
};

__constant__ ImplTab<double, 0> c_d0;
__constant__ ImplTab<double, 1> c_d1;
__constant__ ImplTab<double, 2> c_d2;
__constant__ ImplTab<double, 3> c_d3;
__constant__ ImplTab<float, 0> c_f0;
__constant__ ImplTab<float, 1> c_f1;
__constant__ ImplTab<float, 2> c_f2;
__constant__ ImplTab<float, 3> c_f3;

template <typename T, int P> __device__ __forceinline__ const ImplTab<T, P> &itab();
template <> __device__ __forceinline__ const ImplTab<double, 0> &itab<double, 0>() { return c_d0; }
template <> __device__ __forceinline__ const ImplTab<double, 1> &itab<double, 1>() { return c_d1; }
template <> __device__ __forceinline__ const ImplTab<double, 2> &itab<double, 2>() { return c_d2; }
template <> __device__ __forceinline__ const ImplTab<double, 3> &itab<double, 3>() { return c_d3; }
template <> __device__ __forceinline__ const ImplTab<float, 0> &itab<float, 0>() { return c_f0; }
template <> __device__ __forceinline__ const ImplTab<float, 1> &itab<float, 1>() { return c_f1; }
template <> __device__ __forceinline__ const ImplTab<float, 2> &itab<float, 2>() { return c_f2; }
template <> __device__ __forceinline__ const ImplTab<float, 3> &itab<float, 3>() { return c_f3; }

template <typename T, int P> const void *itab_symbol();
template <> const void *itab_symbol<double, 0>() { return (const void *)&c_d0; }
template <> const void *itab_symbol<double, 1>() { return (const void *)&c_d1; }
template <> const void *itab_symbol<double, 2>() { return (const void *)&c_d2; }
template <> const void *itab_symbol<double, 3>() { return (const void *)&c_d3; }
template <> const void *itab_symbol<float, 0>() { return (const void *)&c_f0; }
template <> const void *itab_symbol<float, 1>() { return (const void *)&c_f1; }
template <> const void *itab_symbol<float, 2>() { return (const void *)&c_f2; }
template <> const void *itab_symbol<float, 3>() { return (const void *)&c_f3; }

template <typename T> struct ImplArgs {
  int K, Kp, nTerms;
  const T *F, *Vn, *rhs;
  const int *nbr, *code;
  const T *A;          // N^2 x Kp: cDot's local part (volume term and own outflow, mass solve applied)
  double gco[4];       // g_m(t) of the source terms
};

// Coefficient `row` of cDot(x)'s parts for element k, by the block's N warps together (row = the warp,
// element = the lane):
//   LOCAL: the local part, the row of the element's matrix (volume term and own outflow, hatM^-1
//          applied), 6 multiply-adds at p = 2 and 10 at p = 3 where the quadrature form of the whole
//          element has 180 and 1600;
//   minus the inflow terms, the part that couples elements: the warps share the 3 R edge points
//          (trace of the neighbour times the velocity, into fl), then every row adds its test functions.
// Contains a block barrier.
template <typename T, int P> struct EdgePoints {   // a warp's edge points, all loads in flight together
  static constexpr int M = (3 * IDims<P>::R + IDims<P>::N - 1) / IDims<P>::N;
  int code, nb[M];
  T v[M];
  __device__ __forceinline__ void load(const ImplArgs<T> &a, int k, bool act) {
    code = act ? a.code[k] : 0;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const int pt = threadIdx.y + i * IDims<P>::N;
      const bool use = act && pt < 3 * IDims<P>::R;
      nb[i] = use ? a.nbr[(size_t)(pt / IDims<P>::R) * a.Kp + k] : -1;
      v[i] = use ? a.Vn[(size_t)pt * a.Kp + k] : T(0);
    }
  }
};
template <typename T, int P, bool LOCAL>
__device__ __forceinline__ T cdot_row(const ImplArgs<T> &a, const EdgePoints<T, P> &ep, const T *x, int k, bool act,
                                      T (*fl)[kRows]) {
  constexpr int N = IDims<P>::N, R = IDims<P>::R;
  const ImplTab<T, P> &tb = itab<T, P>();
  const size_t Kp = a.Kp;
  const int lane = threadIdx.x, row = threadIdx.y;
#pragma unroll
  for (int i = 0; i < EdgePoints<T, P>::M; ++i) {
    const int pt = row + i * N;
    if (pt >= 3 * R) break;
    const int n = pt / R, r = pt - n * R;
    T f = T(0);
    if (ep.v[i] < T(0) && ep.nb[i] >= 0) {
      const T *th = tb.thetaPhi[n][(ep.code >> (2 * n)) & 3][r];
      T tr = T(0);
#pragma unroll
      for (int j = 0; j < N; ++j) tr = fma(th[j], x[j * Kp + ep.nb[i]], tr);
      f = ep.v[i] * tr;
    }
    fl[pt][lane] = f;
  }
  T s = T(0);
  if (LOCAL && act) {
#pragma unroll
    for (int j = 0; j < N; ++j) s = fma(a.A[(size_t)(row * N + j) * Kp + k], x[j * Kp + k], s);
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < 3; ++n)
#pragma unroll
    for (int r = 0; r < R; ++r) s = fma(-tb.Fphi[n][r][row], fl[n * R + r][lane], s);
  return s;
}

// y = ca x + cb cDot(x), cDot with the source terms M^-1 sum_m g_m rhs_m [RHS].
template <typename T, int P, bool RHS>
__global__ void __launch_bounds__(kRows * IDims<P>::N) k_impl_op(const ImplArgs<T> a, const T *__restrict__ x,
                                                                 T *__restrict__ y, double ca, double cb) {
  constexpr int N = IDims<P>::N;
  __shared__ T fl[3 * IDims<P>::R][kRows];
  const int k = blockIdx.x * kRows + threadIdx.x, row = threadIdx.y;
  const size_t Kp = a.Kp;
  const bool act = k < a.K;
  EdgePoints<T, P> ep;
  ep.load(a, k, act);
  T s = cdot_row<T, P, true>(a, ep, x, k, act, fl);
  if (!act) return;
  if (RHS) {
    for (int m = 0; m < a.nTerms; ++m) {
      T q = T(0);
#pragma unroll
      for (int j = 0; j < N; ++j) q = fma(itab<T, P>().hatMinv[row][j], a.rhs[(size_t)(m * N + j) * Kp + k], q);
      s = fma(T(a.gco[m]), q, s);
    }
  }
  y[row * Kp + k] = T(ca) * x[row * Kp + k] + T(cb) * s;
}

// Inverse of each element's diagonal block of y = ca x + cb cDot(x) (volume term and the
// element's own outflow; the neighbours' inflow is off-diagonal), by Gauss-Jordan elimination
// with partial pivoting in FP64.  A block that is singular to the stored type's rounding (a pivot below
// N eps of its largest entry) is replaced by the identity; *inexact is set then, and where the block
// times the stored inverse is off the identity by more than sqrt(eps).  Aloc receives cDot's
// local part itself.
template <typename T, int P>
__global__ void __launch_bounds__(kImplBlock) k_impl_block(const ImplArgs<T> a, double ca, double cb,
                                                           T *__restrict__ Pinv, T *__restrict__ Aloc,
                                                           int *__restrict__ inexact) {
  constexpr int N = IDims<P>::N, Q = IDims<P>::Q, R = IDims<P>::R;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.K) return;
  const ImplTab<T, P> &tb = itab<T, P>();
  const size_t Kp = a.Kp;
  double J[N][N];   // J[i][j]: local part of cDot for c = e_j, before the mass solve
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) J[i][j] = 0.0;
  for (int q = 0; q < Q; ++q) {
    const double f1 = (double)a.F[q * Kp + k], f2 = (double)a.F[(Q + q) * Kp + k];
    for (int j = 0; j < N; ++j) {
      const double pj = (double)tb.phiQ[q][j];
#pragma unroll
      for (int i = 0; i < N; ++i) J[i][j] += ((double)tb.g1[q][i] * f1 + (double)tb.g2[q][i] * f2) * pj;
    }
  }
  const int code = a.code[k];
  for (int n = 0; n < 3; ++n) {
    if (!((code >> (6 + n)) & 1)) continue;
    for (int r = 0; r < R; ++r) {
      const double v = (double)a.Vn[(n * R + r) * Kp + k];
      if (!(v > 0.0)) continue;
      for (int j = 0; j < N; ++j) {
        const double pj = (double)tb.phi1D[n][r][j];
#pragma unroll
        for (int i = 0; i < N; ++i) J[i][j] -= (double)tb.phi1D[n][r][i] * v * pj;
      }
    }
  }
  constexpr double eps = sizeof(T) == 4 ? 0x1p-24 : 0x1p-53, rootEps = sizeof(T) == 4 ? 0x1p-12 : 0x1p-26;
  double A[N][2 * N], most = 0.0;
  for (int i = 0; i < N; ++i) {
    for (int j = 0; j < N; ++j) {
      double s = 0.0;
      for (int l = 0; l < N; ++l) s += (double)tb.hatMinv[i][l] * J[l][j];
      Aloc[(size_t)(i * N + j) * Kp + k] = T(s);
      A[i][j] = (i == j ? ca : 0.0) + cb * s;
      A[i][N + j] = i == j ? 1.0 : 0.0;
      most = fmax(most, fabs(A[i][j]));
    }
  }
  bool ok = true;
  for (int col = 0; col < N && ok; ++col) {
    int piv = col;
    for (int r = col + 1; r < N; ++r)
      if (fabs(A[r][col]) > fabs(A[piv][col])) piv = r;
    if (!(fabs(A[piv][col]) > N * eps * most)) { ok = false; break; }
    if (piv != col)
      for (int j = 0; j < 2 * N; ++j) { const double t = A[col][j]; A[col][j] = A[piv][j]; A[piv][j] = t; }
    const double inv = 1.0 / A[col][col];
    for (int j = 0; j < 2 * N; ++j) A[col][j] *= inv;
    for (int r = 0; r < N; ++r) {
      if (r == col) continue;
      const double f = A[r][col];
      if (f != 0.0)
        for (int j = 0; j < 2 * N; ++j) A[r][j] -= f * A[col][j];
    }
  }
  double off = 0.0;             // of the block, as it is applied, times the inverse, as it is stored
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      double s = i == j ? -1.0 : 0.0;
      for (int l = 0; l < N; ++l)
        s += ((i == l ? ca : 0.0) + cb * (double)Aloc[(size_t)(i * N + l) * Kp + k]) * (double)T(A[l][N + j]);
      off = fmax(off, fabs(s));
      ok = ok && isfinite(s);
    }
  if (!ok || off > rootEps) *inexact = 1;
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) Pinv[(i * N + j) * Kp + k] = T(ok ? A[i][N + j] : (i == j ? 1.0 : 0.0));
}

// ---- vector kernels over n = N Kp values ------------------------------------------------------

// A sum over the grid in a fixed order: every block adds its threads' shares, group after group of 32
// elements, the block that arrives last adds the blocks' (in block order, whichever block it is).
// kSumBlocks blocks at most, as many as the SMs hold at a time, so that this last addition stays short
// beside the kernel: with a block per group, one block was left K / 32 shares of every basis vector
// (524288 triangles, an Arnoldi step in FP64: p = 1 905 us so and 397 now, p = 2 1361 and 768; 32768
// triangles, 1024 groups either way, 78 and 83 us).
constexpr int kSumBlocks = 8 * 152;
struct GridSums {
  double *partial;          // vector v, block b at v * gridDim.x + b
  unsigned int *ticket;     // blocks that have stored their shares (0 between launches)
  double *out;
};
// Sums x[0 .. n) over a warp's lanes, in every lane.  On the integer units: each share rounded to 57 bits
// below the lanes' largest exponent (off by at most 2^-58 of it, and no share one way, where each FP64
// addition rounds at 2^-53), one redux and five exchanges and additions of 64-bit words, n sums side by side; five FP64
// additions each would hold the warp's scheduler for 380 cycles.  Shares outside 2^(+-800) take the
// FP64 form.
template <int n> __device__ __forceinline__ void warp_sums(double x[n]) {
  int E[n];
  bool ok = true;
#pragma unroll
  for (int q = 0; q < n; ++q) {
    E[q] = __reduce_max_sync(0xffffffffu, __double2hiint(x[q]) & 0x7fffffff) >> 20;
    ok = ok && (E[q] == 0 || (E[q] >= 223 && E[q] <= 1823));
  }
  if (!ok) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < n; ++q) x[q] += __shfl_xor_sync(0xffffffffu, x[q], o);
    return;
  }
  long long v[n];
#pragma unroll
  for (int q = 0; q < n; ++q) v[q] = fx::fix_near<57>(x[q], max(E[q], 223));   // all zero: zero
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < n; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
#pragma unroll
  for (int q = 0; q < n; ++q) x[q] = fx::to_double_int(v[q], max(E[q], 223) - 1022 - 57);
}
// The threads' shares x[0 .. n) of vectors v0 ...: added over the block into tot (the block's sums, set by its
// first group).
constexpr int kMaxSums = 258;
template <int N>
__device__ __forceinline__ void add_shares(double *tot, bool first, int v0, int n, double x[kVecs]) {
  __shared__ double sh[N][kVecs];
  __syncthreads();                            // the shares before are read
  if (n <= 2) warp_sums<2>(x);                // the values beyond n are zero
  else if (n <= 4) warp_sums<4>(x);
  else warp_sums<kVecs>(x);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < kVecs; ++q) sh[threadIdx.y][q] = x[q];
  __syncthreads();
  if (threadIdx.y == 0 && (int)threadIdx.x < n) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) s += sh[i][threadIdx.x];
    tot[v0 + threadIdx.x] = first ? s : tot[v0 + threadIdx.x] + s;   // always this thread's
  }
}
// After the shares of nv vectors: the last block writes their sums.
template <int N>
__device__ __forceinline__ void finish_sums(const GridSums &gs, const double *tot, int nv) {
  __shared__ bool last;
  __syncthreads();
  for (int v = threadIdx.y * 32 + threadIdx.x; v < nv; v += 32 * N) gs.partial[(size_t)v * gridDim.x + blockIdx.x] = tot[v];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) last = atomicAdd(gs.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  constexpr int kV = 2;                       // vectors of a warp at once
  for (int v0 = kV * threadIdx.y; v0 < nv; v0 += kV * N) {
    double s[kV] = {0.0, 0.0};
#pragma unroll 8
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32)
#pragma unroll
      for (int q = 0; q < kV; ++q)
        if (v0 + q < nv) s[q] += __ldcg(&gs.partial[(size_t)(v0 + q) * gridDim.x + b]);
    warp_sums<kV>(s);
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < kV; ++q)
        if (v0 + q < nv) gs.out[v0 + q] = s[q];
  }
  if (threadIdx.x == 0 && threadIdx.y == 0) *gs.ticket = 0;
}
// The shares of <V_v, y> for v < nv, at = row Kp + k the thread's place (inactive: y = 0, at within V).
template <typename T, int N>
__device__ __forceinline__ void share_products(double *tot, bool first, const T *V, size_t n, size_t at, int nv, double y) {
  for (int v0 = 0; v0 < nv; v0 += kVecs) {
    double s[kVecs];
#pragma unroll
    for (int q = 0; q < kVecs; ++q) s[q] = v0 + q < nv ? (double)V[(size_t)(v0 + q) * n + at] : 0.0;
#pragma unroll
    for (int q = 0; q < kVecs; ++q) s[q] *= y;
    add_shares<N>(tot, first, v0, min(kVecs, nv - v0), s);
  }
}
// y + sgn sum_{v < nv} h_v V_v at the thread's place
template <typename T>
__device__ __forceinline__ double add_vectors(const T *V, size_t n, size_t at, int nv, const double *h, double sgn,
                                              double y) {
  for (int v0 = 0; v0 < nv; v0 += kVecs) {
    double a[kVecs];
#pragma unroll
    for (int q = 0; q < kVecs; ++q) a[q] = v0 + q < nv ? (double)V[(size_t)(v0 + q) * n + at] : 0.0;
#pragma unroll
    for (int q = 0; q < kVecs; ++q)
      if (v0 + q < nv) y += sgn * h[v0 + q] * a[q];
  }
  return y;
}
// Row `row` of P^-1 v for the block's elements, v given a value per thread.  Contains a block barrier.
template <typename T, int N>
__device__ __forceinline__ T precondition_row(const T *Pinv, size_t Kp, int k, bool act, T v, T (*vs)[kRows]) {
  vs[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  T s = T(0);
  if (act) {
#pragma unroll
    for (int j = 0; j < N; ++j) s = fma(Pinv[(size_t)(threadIdx.y * N + j) * Kp + k], vs[j][threadIdx.x], s);
  }
  return s;
}

// y = sum_v c_v x_v (host coefficients, up to kChunk vectors; y may alias an input)
template <typename T> struct Comb {
  const T *x[kChunk];
  double c[kChunk];
  int nv;
};
template <typename T>
__global__ void __launch_bounds__(kVecThreads) k_comb(T *y, const Comb<T> cb, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    double s = 0.0;
#pragma unroll
    for (int v = 0; v < kChunk; ++v)
      if (v < cb.nv) s += cb.c[v] * (double)cb.x[v][i];
    y[i] = T(s);
  }
}

// The small dense part of GMRES: Hessenberg matrix, Givens rotations, residual estimate.
// status: [0] |g_{j+1}|, [1] columns in use, [2] breakdown seen (later columns are ignored).
struct GmresDense {
  double *H, *cs, *sn, *g, *y, *status;   // H: (m + 1) x m, column-major
};

// One Arnoldi step is three kernels over the elements (it was eleven launches and 90 us at 8192
// elements, p = 2; now about 40 us):
//   k_arn_apply   w = A P^-1 v_j; h1 = V^T w.  z = P^-1 v_j comes from the step before.  P inverts the
//                 element's own block of A, so the local part of A z is v_j itself and only the
//                 neighbours' inflow is left (IDENT; a mesh with a block whose stored inverse is off, or
//                 singular with the identity in its place, applies the whole operator)
//   k_arn_first   w -= V h1; h2 = V^T w and |w|^2        (classical Gram-Schmidt, second pass)
//   k_arn_second  w -= V h2; v_{j+1} = w / |w|, with |w|^2 after the pass from |w|^2 - |h2|^2 (h2 is at
//                 rounding level beside w, until the Krylov space is used up and the residual is there too);
//                 z = P^-1 v_{j+1}; column j of the Hessenberg matrix and the Givens rotations in one more
//                 block
template <typename T, int P, bool IDENT>
__global__ void __launch_bounds__(kRows * IDims<P>::N)
k_arn_apply(const ImplArgs<T> a, const T *__restrict__ V, size_t n, int j, const T *__restrict__ z, T *__restrict__ w,
            double ca, double cb, const GridSums gs) {
  constexpr int N = IDims<P>::N;
  __shared__ T fl[3 * IDims<P>::R][kRows];
  __shared__ double tot[kMaxSums];
  for (int grp = blockIdx.x; grp * kRows < a.K; grp += gridDim.x) {
    const int k = grp * kRows + threadIdx.x;
    const bool act = k < a.K;
    const size_t at = (size_t)threadIdx.y * a.Kp + (act ? k : 0);
    EdgePoints<T, P> ep;
    ep.load(a, k, act);
    const T s = cdot_row<T, P, !IDENT>(a, ep, z, k, act, fl);
    T y = T(0);
    if (act) {
      y = (IDENT ? V[(size_t)j * n + at] : T(ca) * z[at]) + T(cb) * s;
      w[at] = y;
    }
    share_products<T, N>(tot, grp == (int)blockIdx.x, V, n, at, j + 1, (double)y);
  }
  finish_sums<N>(gs, tot, j + 1);
}

template <typename T, int N>
__global__ void __launch_bounds__(kRows * N) k_arn_first(int K, int Kp, const T *V, size_t n, int j, T *w,
                                                         const double *h1, const GridSums gs) {
  __shared__ double sh[257], tot[kMaxSums];
  for (int v = threadIdx.y * 32 + threadIdx.x; v <= j; v += 32 * N) sh[v] = h1[v];
  __syncthreads();
  for (int grp = blockIdx.x; grp * kRows < K; grp += gridDim.x) {
    const int k = grp * kRows + threadIdx.x;
    const bool act = k < K, first = grp == (int)blockIdx.x;
    const size_t at = (size_t)threadIdx.y * Kp + (act ? k : 0);
    double y = act ? (double)w[at] : 0.0;
    if (act) {
      const T t = T(add_vectors(V, n, at, j + 1, sh, -1.0, y));
      w[at] = t;
      y = (double)t;
    }
    share_products<T, N>(tot, first, V, n, at, j + 1, y);
    double s[kVecs] = {y * y};
    add_shares<N>(tot, first, j + 1, 1, s);
  }
  finish_sums<N>(gs, tot, j + 2);
}

// Column j: h1 + h2, the earlier rotations, a new one, the residual estimate.  One warp; the chain of
// rotations runs on one lane from shared memory.
__device__ __forceinline__ void gmres_column(const GmresDense &d, const double *h1, const double *h2, double nrm2, int j,
                                             int m, double *col, double *cs, double *sn) {
  const int l = threadIdx.x;
  for (int i = l; i <= j; i += 32) {
    col[i] = h1[i] + h2[i];
    if (i < j) { cs[i] = d.cs[i]; sn[i] = d.sn[i]; }
  }
  __syncwarp();
  if (l == 0 && d.status[2] == 0.0) {
    double c0 = col[0];
    for (int i = 0; i < j; ++i) {
      const double c1 = col[i + 1];
      col[i] = cs[i] * c0 + sn[i] * c1;
      c0 = -sn[i] * c0 + cs[i] * c1;
    }
    const double nw = sqrt(fmax(nrm2, 0.0));
    const double r = hypot(c0, nw);
    const double c = r > 0.0 ? c0 / r : 1.0, s = r > 0.0 ? nw / r : 0.0;
    d.cs[j] = c;
    d.sn[j] = s;
    col[j] = r;
    const double g = d.g[j];
    d.g[j + 1] = -s * g;
    d.g[j] = c * g;
    d.status[0] = fabs(s * g);
    d.status[1] = (double)(j + 1);
    if (r == 0.0) d.status[2] = 1.0;
    cs[0] = 1.0;   // the column counts
  } else if (l == 0) {
    cs[0] = 0.0;
  }
  __syncwarp();
  if (cs[0] != 0.0)
    for (int i = l; i <= j; i += 32) d.H[(size_t)j * (m + 1) + i] = col[i];
  if (l == 0 && cs[0] != 0.0) d.H[(size_t)j * (m + 1) + j + 1] = 0.0;
}

// h2: then |w|^2 at j + 1.  The last block has no elements: the column.
template <typename T, int N>
__global__ void __launch_bounds__(kRows * N)
k_arn_second(int K, int Kp, T *V, size_t n, int j, const T *w, const T *__restrict__ Pinv, T *z, const double *h1,
             const double *h2, GmresDense d, int m) {
  __shared__ double col[257], cs[257], sn[257];
  __shared__ double norm;
  __shared__ T vs[N][kRows];
  const int k = blockIdx.x * kRows + threadIdx.x;
  const bool act = blockIdx.x != gridDim.x - 1 && k < K;
  T pr[N];                  // the row of P^-1, in flight with the rest
#pragma unroll
  for (int i = 0; i < N; ++i) pr[i] = act ? Pinv[(size_t)(threadIdx.y * N + i) * Kp + k] : T(0);
  if (threadIdx.y == 0) {   // |w|^2 - |h2|^2
    double q[1] = {0.0};
    for (int v = threadIdx.x; v <= j; v += 32) {
      col[v] = h2[v];
      q[0] += col[v] * col[v];
    }
    warp_sums<1>(q);
    if (threadIdx.x == 0) norm = h2[j + 1] - q[0];
  }
  const size_t at = (size_t)threadIdx.y * Kp + (act ? k : 0);
  double y = act ? (double)w[at] : 0.0;
  __syncthreads();
  const double nrm2 = norm;
  if (blockIdx.x == gridDim.x - 1) {
    if (threadIdx.y == 0) gmres_column(d, h1, h2, nrm2, j, m, col, cs, sn);
    return;
  }
  const double s = nrm2 > 0.0 ? 1.0 / sqrt(nrm2) : 0.0;
  T v1 = T(0);
  if (act) {
    v1 = T(add_vectors(V, n, at, j + 1, col, -1.0, y) * s);
    V[(size_t)(j + 1) * n + at] = v1;
  }
  vs[threadIdx.y][threadIdx.x] = v1;
  __syncthreads();
  T zz = T(0);
#pragma unroll
  for (int i = 0; i < N; ++i) zz = fma(pr[i], vs[i][threadIdx.x], zz);
  if (act) z[at] = zz;
}

// r = b - (ca x + cb cDot(x)), gs.out[0] = |r|^2, [1] = |b|^2
template <typename T, int P>
__global__ void __launch_bounds__(kRows * IDims<P>::N)
k_impl_residual(const ImplArgs<T> a, const T *__restrict__ b, const T *__restrict__ x, T *__restrict__ r, double ca,
                double cb, const GridSums gs) {
  constexpr int N = IDims<P>::N;
  __shared__ T fl[3 * IDims<P>::R][kRows];
  __shared__ double tot[2];
  for (int grp = blockIdx.x; grp * kRows < a.K; grp += gridDim.x) {
    const int k = grp * kRows + threadIdx.x;
    const bool act = k < a.K;
    const size_t at = (size_t)threadIdx.y * a.Kp + (act ? k : 0);
    EdgePoints<T, P> ep;
    ep.load(a, k, act);
    const T s = cdot_row<T, P, true>(a, ep, x, k, act, fl);
    double q[kVecs] = {0.0};
    if (act) {
      const T bi = b[at], y = T(ca) * x[at] + T(cb) * s, ri = T((double)bi - (double)y);
      r[at] = ri;
      q[0] = (double)ri * (double)ri;
      q[1] = (double)bi * (double)bi;
    }
    add_shares<N>(tot, grp == (int)blockIdx.x, 0, 2, q);
  }
  finish_sums<N>(gs, tot, 2);
}

// v_0 = r / |r|, z = P^-1 v_0, and the dense part of a new cycle.
template <typename T, int N>
__global__ void __launch_bounds__(kRows * N) k_arn_start(int K, int Kp, const T *__restrict__ r, T *__restrict__ V,
                                                         const T *__restrict__ Pinv, T *__restrict__ z,
                                                         const double *__restrict__ nrm2, GmresDense d, int m) {
  __shared__ T vs[N][kRows];
  const int k = blockIdx.x * kRows + threadIdx.x;
  const bool act = k < K;
  const size_t at = (size_t)threadIdx.y * Kp + (act ? k : 0);
  const double nr = nrm2[0];
  if (blockIdx.x == 0 && threadIdx.y == 0) {
    for (int i = threadIdx.x; i <= m; i += 32) d.g[i] = i == 0 ? sqrt(fmax(nr, 0.0)) : 0.0;
    if (threadIdx.x == 0) { d.status[0] = sqrt(fmax(nr, 0.0)); d.status[1] = 0.0; d.status[2] = 0.0; }
  }
  T v = T(0);
  if (act) {
    v = T((double)r[at] * (nr > 0.0 ? 1.0 / sqrt(nr) : 0.0));
    V[at] = v;
  }
  const T zz = precondition_row<T, N>(Pinv, Kp, k, act, v, vs);
  if (act) z[at] = zz;
}

// y = H^-1 g over the columns in use (upper triangular), zero beyond them.  The columns come to shared
// memory first (up to kSolveCols of them); then one warp takes each solved unknown off the rows
// above it, the lanes side by side.
constexpr int kSolveCols = 64;
__global__ void k_gmres_solve(GmresDense d, int m) {
  __shared__ double g[256], H[kSolveCols * (kSolveCols + 1)];
  const int je = (int)d.status[1], l = threadIdx.x;
  const bool held = je <= kSolveCols;
  for (int i = l; i < m; i += blockDim.x) {
    if (i < je) g[i] = d.g[i];
    else d.y[i] = 0.0;
  }
  if (held)
    for (int e = l; e < je * je; e += blockDim.x) {
      const int c = e / je, r = e - c * je;
      H[c * (kSolveCols + 1) + r] = d.H[(size_t)c * (m + 1) + r];
    }
  __syncthreads();
  if (l >= 32) return;
  for (int i = je - 1; i >= 0; --i) {
    const double *col = held ? &H[i * (kSolveCols + 1)] : &d.H[(size_t)i * (m + 1)];
    const double y = col[i] != 0.0 ? g[i] / col[i] : 0.0;
    for (int q = l; q < i; q += 32) g[q] -= col[q] * y;
    if (l == 0) d.y[i] = y;
    __syncwarp();
  }
}

// x += P^-1 V y over nv vectors
template <typename T, int N>
__global__ void __launch_bounds__(kRows * N) k_arn_update(int K, int Kp, const T *__restrict__ V, size_t n, int nv,
                                                          const double *__restrict__ y, const T *__restrict__ Pinv,
                                                          T *__restrict__ x) {
  __shared__ T vs[N][kRows];
  const int k = blockIdx.x * kRows + threadIdx.x;
  const bool act = k < K;
  const size_t at = (size_t)threadIdx.y * Kp + (act ? k : 0);
  const T t = act ? T(add_vectors(V, n, at, nv, y, 1.0, 0.0)) : T(0);
  const T z = precondition_row<T, N>(Pinv, Kp, k, act, t, vs);
  if (act) x[at] = T((double)x[at] + (double)z);
}

double time_factor_of(int fn, double t) { return fn == DGADV_TIME_EXP_NEG ? std::exp(-t) : 1.0; }

// DIRK tables (core/rungeKuttaImplicit.m); returns the number of stages.
int dirk_table(int ord, double a[5][5]) {
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < 5; ++j) a[i][j] = 0.0;
  switch (ord) {
    case 1: a[0][0] = 1.0; return 1;
    case 2: {
      const double l = 0.5 * (2.0 - std::sqrt(2.0));
      a[0][0] = l; a[1][0] = 1.0 - l; a[1][1] = l;
      return 2;
    }
    case 3: {
      const double al = 0.4358665215084589994160194511935568425292;
      const double be = 0.5 * (1. + al);
      const double b1 = -0.25 * (6 * al * al - 16 * al + 1);
      const double b2 = 0.25 * (6 * al * al - 20 * al + 5);
      a[0][0] = al; a[1][0] = be - al; a[1][1] = al; a[2][0] = b1; a[2][1] = b2; a[2][2] = al;
      return 3;
    }
    case 4: {
      const double g = 1. / 4.;
      const double t[5][5] = {{g, 0, 0, 0, 0},
                              {1. / 2., g, 0, 0, 0},
                              {17. / 50., -1. / 25., g, 0, 0},
                              {371. / 1360., -137. / 2720., 15. / 544., g, 0},
                              {25. / 24., -49. / 48., 125. / 16., -85. / 12., g}};
      for (int i = 0; i < 5; ++i)
        for (int j = 0; j < 5; ++j) a[i][j] = t[i][j];
      return 5;
    }
  }
  return 0;
}

}  // namespace

// Solver state of a handle: Krylov basis, work vectors, preconditioner, scratch.
struct ImplicitState {
  int m = 0;                      // restart length
  size_t n = 0;                   // N * Kp
  void *V = nullptr;              // (m + 1) x n
  void *w = nullptr, *z = nullptr, *r = nullptr, *x = nullptr, *b = nullptr, *zero = nullptr, *s = nullptr;
  void *kst = nullptr;            // 4 x n stage derivatives
  void *Pinv = nullptr;           // N^2 x Kp
  double pinvA = 0.0, pinvB = 0.0;
  int pinvVersion = -1;           // velocity version the blocks were built for
  void *Aloc = nullptr;           // N^2 x Kp: cDot's local part
  int *inexact = nullptr;         // a diagonal block was singular, or its stored inverse is off
  bool ident = false;             // ... none was: P^-1 inverts every diagonal block
  int blocks = 0;                 // the element kernels' blocks: one per group of 32
  int sumBlocks = 0;              // ... of those that add over the grid
  double *partial = nullptr;      // (m + 2) x sumBlocks
  unsigned int *ticket = nullptr;
  double *dres = nullptr;         // h1 (m + 1), h2 and |w|^2 (m + 2)
  double *dense = nullptr;        // H ((m + 1) x m), cs, sn, g, y, status
  std::vector<cudaGraphExec_t> arnoldi;   // Arnoldi step j as a CUDA graph, for (graphA, graphB)
  double graphA = 0.0, graphB = 0.0;
  double *hres = nullptr;         // pinned mirror of dres
  bool tablesLoaded = false;
};

void implicit_release(dgadv_handle *h) {
  ImplicitState *st = h->impl;
  if (!st) return;
  for (cudaGraphExec_t g : st->arnoldi)
    if (g) cudaGraphExecDestroy(g);
  if (st->hres) cudaFreeHost(st->hres);
  delete st;   // device buffers belong to h->allocs
  h->impl = nullptr;
}

namespace {

template <typename T, int P>
cudaError_t upload_itab(const RefTables &rt, cudaStream_t stream) {
  using I = IDims<P>;
  static ImplTab<T, P> t;   // host staging (the async copy reads it later on the stream)
  if (rt.Q != I::Q || rt.R != I::R || rt.N != I::N) return cudaErrorInvalidValue;
  for (int q = 0; q < I::Q; ++q)
    for (int i = 0; i < I::N; ++i) {
      t.phiQ[q][i] = T(rt.phiQ[q * I::N + i]);
      t.g1[q][i] = T(rt.gradQ[q * I::N + i]);
      t.g2[q][i] = T(rt.gradQ[I::Q * I::N + q * I::N + i]);
    }
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < I::R; ++r)
      for (int i = 0; i < I::N; ++i) {
        t.phi1D[n][r][i] = T(rt.phi1D[(n * I::R + r) * I::N + i]);
        for (int np = 0; np < 3; ++np)
          t.thetaPhi[n][np][r][i] = T(rt.thetaPhi[((n * 3 + np) * I::R + r) * I::N + i]);
      }
  for (int i = 0; i < I::N; ++i)
    for (int j = 0; j < I::N; ++j) t.hatMinv[i][j] = T(rt.hatMinv[i * I::N + j]);
  for (int n = 0; n < 3; ++n)
    for (int r = 0; r < I::R; ++r)
      for (int i = 0; i < I::N; ++i) {
        double a = 0.0;
        for (int j = 0; j < I::N; ++j) a += rt.hatMinv[i * I::N + j] * rt.phi1D[(n * I::R + r) * I::N + j];
        t.Fphi[n][r][i] = T(a);
      }
  const cudaError_t e = cudaMemcpyToSymbolAsync(itab_symbol<T, P>(), &t, sizeof(t), 0, cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(stream);
}

template <typename T, int P>
struct Solver {
  dgadv_handle *h;
  ImplicitState *st;
  ImplArgs<T> args;
  size_t n;
  int gridV;
  static constexpr int N = IDims<P>::N;

  explicit Solver(dgadv_handle *hh) : h(hh), st(hh->impl) {
    n = st->n;
    args = ImplArgs<T>{};
    args.K = h->K; args.Kp = h->Kp; args.nTerms = h->nTerms;
    args.F = (const T *)h->F; args.Vn = (const T *)h->Vn; args.rhs = (const T *)h->rhs;
    args.nbr = h->nbr; args.code = h->code; args.A = (const T *)st->Aloc;
    gridV = (int)std::min<size_t>((n + kVecThreads - 1) / kVecThreads, 4 * 152);
  }
  T *vec(void *p) const { return (T *)p; }
  T *basis(int j) const { return (T *)st->V + (size_t)j * n; }
  GridSums sums(double *out) const { return GridSums{st->partial, st->ticket, out}; }

  // y = ca x + cb cDot(x; t) (sources if withRhs)
  void op(const T *x, T *y, double ca, double cb, bool withRhs, double t) {
    ImplArgs<T> a = args;
    const bool rhs = withRhs && h->nTerms > 0 && h->rhs;
    for (int m = 0; m < h->nTerms; ++m) a.gco[m] = time_factor_of(h->timeFn[m], t);
    if (rhs) k_impl_op<T, P, true><<<st->blocks, dim3(kRows, N), 0, h->stream>>>(a, x, y, ca, cb);
    else k_impl_op<T, P, false><<<st->blocks, dim3(kRows, N), 0, h->stream>>>(a, x, y, ca, cb);
  }
  // The diagonal blocks' inverses and cDot's local part, whenever the velocity or the stage's
  // coefficients changed.
  int build_prec(double ca, double cb) {
    if (st->pinvVersion == h->velVersion && st->pinvA == ca && st->pinvB == cb) return DGADV_OK;
    int inexact = 0;
    DG_CUDA(cudaMemsetAsync(st->inexact, 0, sizeof(int), h->stream));
    k_impl_block<T, P><<<st->blocks, kRows, 0, h->stream>>>(args, ca, cb, (T *)st->Pinv, (T *)st->Aloc, st->inexact);
    DG_CUDA(cudaMemcpyAsync(&inexact, st->inexact, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    DG_CUDA(cudaStreamSynchronize(h->stream));
    if (st->ident != (inexact == 0)) st->graphA = st->graphB = 0.0;   // the steps' graphs hold the other kernel
    st->ident = inexact == 0;
    st->pinvA = ca; st->pinvB = cb; st->pinvVersion = h->velVersion;
    return DGADV_OK;
  }
  void comb(T *y, const Comb<T> &cb) { k_comb<T><<<gridV, kVecThreads, 0, h->stream>>>(y, cb, n); }

  // Arnoldi step j: w = A P^-1 v_j, orthogonalised against v_0..v_j (classical Gram-Schmidt,
  // twice), v_{j+1} = w / |w|, z = P^-1 v_{j+1}, and the dense update of column j.
  void arnoldi_enqueue(int j, double ca, double cb, const GmresDense &d) {
    const int m = st->m, nb = st->blocks, ns = st->sumBlocks;
    const dim3 nt(kRows, N);
    T *w = vec(st->w), *z = vec(st->z), *V = basis(0);
    double *h1 = st->dres, *h2 = st->dres + (m + 1);
    if (st->ident) k_arn_apply<T, P, true><<<ns, nt, 0, h->stream>>>(args, V, n, j, z, w, ca, cb, sums(h1));
    else k_arn_apply<T, P, false><<<ns, nt, 0, h->stream>>>(args, V, n, j, z, w, ca, cb, sums(h1));
    k_arn_first<T, N><<<ns, nt, 0, h->stream>>>(h->K, h->Kp, V, n, j, w, h1, sums(h2));
    k_arn_second<T, N><<<nb + 1, nt, 0, h->stream>>>(h->K, h->Kp, V, n, j, w, (const T *)st->Pinv, z, h1, h2, d, m);
  }
  // Steps j .. j + cnt - 1: kCheck of them, between two looks at the residual, as one CUDA graph captured
  // once per j and operator (all its buffers are the handle's own; the operator's coefficients are
  // baked in); fewer are launched directly.
  int arnoldi_steps(int j, int cnt, double ca, double cb, const GmresDense &d) {
    if ((h->flags & DGADV_FLAG_NO_GRAPH) || cnt != kCheck) {
      for (int i = 0; i < cnt; ++i) arnoldi_enqueue(j + i, ca, cb, d);
      return cudaGetLastError() == cudaSuccess ? DGADV_OK : DGADV_ECUDA;
    }
    if (st->graphA != ca || st->graphB != cb || (int)st->arnoldi.size() != st->m) {
      for (cudaGraphExec_t g : st->arnoldi)
        if (g) cudaGraphExecDestroy(g);
      st->arnoldi.assign(st->m, nullptr);
      st->graphA = ca;
      st->graphB = cb;
    }
    if (!st->arnoldi[j]) {
      cudaGraph_t g = nullptr;
      if (cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return DGADV_ECUDA;
      for (int i = 0; i < cnt; ++i) arnoldi_enqueue(j + i, ca, cb, d);
      if (cudaStreamEndCapture(h->stream, &g) != cudaSuccess) return DGADV_ECUDA;
      const cudaError_t e = cudaGraphInstantiate(&st->arnoldi[j], g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return DGADV_ECUDA;
    }
    return cudaGraphLaunch(st->arnoldi[j], h->stream) == cudaSuccess ? DGADV_OK : DGADV_ECUDA;
  }

  // Solves (ca I + cb cDot0) x = b, x holding the initial guess; right block-Jacobi
  // preconditioning.  The Hessenberg column, the Givens rotations and the small triangular
  // solve run on the device; the host reads the residual estimate every kCheck iterations
  // (a few iterations past convergence only improve the iterate).  Returns DGADV_OK or
  // DGADV_ENOCONV; iters accumulates iterations.
  int gmres(const T *b, T *x, double ca, double cb, double tol, int maxIter, int &iters, double &relres) {
    const int m = st->m, nb = st->blocks;
    const dim3 nt(kRows, N);
    if (int e = build_prec(ca, cb)) return e;
    T *z = vec(st->z), *r = vec(st->r);
    GmresDense d;
    d.H = st->dense;
    d.cs = d.H + (size_t)(m + 1) * m;
    d.sn = d.cs + m;
    d.g = d.sn + m;
    d.y = d.g + (m + 1);
    d.status = d.y + m;
    int used = 0;
    for (;;) {
      k_impl_residual<T, P><<<st->sumBlocks, nt, 0, h->stream>>>(args, b, x, r, ca, cb, sums(st->dres));
      cudaMemcpyAsync(st->hres, st->dres, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
      if (cudaStreamSynchronize(h->stream) != cudaSuccess) return DGADV_ECUDA;
      const double bnorm = std::sqrt(st->hres[1]);
      if (bnorm == 0.0) {
        cudaMemsetAsync(x, 0, n * sizeof(T), h->stream);
        relres = 0.0;
        return DGADV_OK;
      }
      relres = std::sqrt(st->hres[0]) / bnorm;
      if (relres <= tol) return DGADV_OK;
      if (used >= maxIter) return DGADV_ENOCONV;
      k_arn_start<T, N><<<nb, nt, 0, h->stream>>>(h->K, h->Kp, r, basis(0), (const T *)st->Pinv, z, st->dres, d, m);
      int j = 0;
      while (j < m && used < maxIter) {
        const int cnt = std::min(std::min(kCheck, m - j), maxIter - used);
        if (int e = arnoldi_steps(j, cnt, ca, cb, d)) return e;
        used += cnt;
        iters += cnt;
        j += cnt;
        cudaMemcpyAsync(st->hres, d.status, 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
        if (cudaStreamSynchronize(h->stream) != cudaSuccess) return DGADV_ECUDA;
        relres = st->hres[0] / bnorm;
        if (relres <= tol || st->hres[2] != 0.0) break;
      }
      // x += P^-1 V y with y = H^-1 g over the columns in use
      k_gmres_solve<<<1, 256, 0, h->stream>>>(d, m);
      k_arn_update<T, N><<<nb, nt, 0, h->stream>>>(h->K, h->Kp, basis(0), n, j, d.y, (const T *)st->Pinv, x);
    }
  }

  int dirk_steps(int nSteps, int nStep0, double tau, int ord, double tol, int maxIter, int &iters,
                 double &worst) {
    double a[5][5];
    const int S = dirk_table(ord, a);
    if (!S) { h->err = "DIRK order must be 1..4"; return DGADV_EINVAL; }
    T *cn = (T *)h->cn, *x = vec(st->x), *rhs = vec(st->b), *s = vec(st->s);
    const T *zero = vec(st->zero);
    const bool sources = h->nTerms > 0 && h->rhs;
    worst = 0.0;
    if (int e = build_prec(1.0, -tau * a[0][0])) return e;   // the operator needs the local part
    for (int nn = 0; nn < nSteps; ++nn) {
      const double t0 = (double)(nStep0 + nn) * tau;
      cudaMemcpyAsync(x, cn, n * sizeof(T), cudaMemcpyDeviceToDevice, h->stream);
      for (int i = 0; i < S; ++i) {
        double ci = 0.0;
        for (int j = 0; j <= i; ++j) ci += a[i][j];
        const double ti = t0 + ci * tau, gam = tau * a[i][i];
        if (sources) op(zero, s, 0.0, 1.0, true, ti);    // s_i = M^-1 sysV(t_i)
        Comb<T> cb{};
        cb.nv = 0;
        cb.x[cb.nv] = cn; cb.c[cb.nv++] = 1.0;
        for (int j = 0; j < i; ++j) { cb.x[cb.nv] = (const T *)st->kst + (size_t)j * n; cb.c[cb.nv++] = tau * a[i][j]; }
        if (sources) { cb.x[cb.nv] = s; cb.c[cb.nv++] = gam; }
        comb(rhs, cb);
        double rr = 0.0;
        const int e = gmres(rhs, x, 1.0, -gam, tol, maxIter, iters, rr);
        worst = std::max(worst, rr);
        if (e) return e;
        if (i + 1 < S) op(x, (T *)st->kst + (size_t)i * n, 0.0, 1.0, true, ti);   // k_i
      }
      cudaMemcpyAsync(cn, x, n * sizeof(T), cudaMemcpyDeviceToDevice, h->stream);
    }
    return cudaStreamSynchronize(h->stream) == cudaSuccess ? DGADV_OK : DGADV_ECUDA;
  }

  int stationary(double tol, int maxIter, int &iters, double &res) {
    T *cn = (T *)h->cn, *s = vec(st->s);
    if (int e = build_prec(0.0, -1.0)) return e;
    op(vec(st->zero), s, 0.0, 1.0, true, 0.0);         // M^-1 sysV
    const int e = gmres(s, cn, 0.0, -1.0, tol, maxIter, iters, res);   // M^-1 A x = M^-1 sysV
    if (e) return e;
    return cudaStreamSynchronize(h->stream) == cudaSuccess ? DGADV_OK : DGADV_ECUDA;
  }
};

int allocate_state(dgadv_handle *h, ImplicitState *st, int restart) {
  const size_t rb = ops_of(h).realBytes;
  st->m = restart;
  st->n = (size_t)h->N * h->Kp;
  const size_t vb = st->n * rb;
  void **bufs[] = {&st->w, &st->z, &st->r, &st->x, &st->b, &st->zero, &st->s};
  int e;
  if ((e = dev_alloc(h, &st->V, (size_t)(restart + 1) * vb))) return e;
  for (void **b : bufs)
    if ((e = dev_alloc(h, b, vb))) return e;
  if ((e = dev_alloc(h, &st->kst, 4 * vb))) return e;
  if ((e = dev_alloc(h, &st->Pinv, (size_t)h->N * h->N * h->Kp * rb))) return e;
  if ((e = dev_alloc(h, &st->Aloc, (size_t)h->N * h->N * h->Kp * rb))) return e;
  st->blocks = (h->K + kRows - 1) / kRows;
  st->sumBlocks = std::min(st->blocks, kSumBlocks);
  if ((e = dev_alloc(h, (void **)&st->partial, (size_t)(restart + 2) * st->sumBlocks * 8))) return e;
  if ((e = dev_alloc(h, (void **)&st->ticket, 16))) return e;
  if ((e = dev_alloc(h, (void **)&st->inexact, 16))) return e;
  if ((e = dev_alloc(h, (void **)&st->dres, (size_t)(2 * restart + 3) * 8))) return e;
  DG_CUDA(cudaMemsetAsync(st->ticket, 0, 16, h->stream));
  if ((e = dev_alloc(h, (void **)&st->dense, ((size_t)(restart + 1) * restart + 4 * (size_t)restart + 8) * 8))) return e;
  DG_CUDA(cudaMallocHost((void **)&st->hres, (size_t)3 * (restart + 1) * 8));
  DG_CUDA(cudaMemsetAsync(st->V, 0, (size_t)(restart + 1) * vb, h->stream));
  for (void **b : bufs) DG_CUDA(cudaMemsetAsync(*b, 0, vb, h->stream));
  DG_CUDA(cudaMemsetAsync(st->kst, 0, 4 * vb, h->stream));
  DG_CUDA(cudaStreamSynchronize(h->stream));
  return DGADV_OK;
}

int ensure_state(dgadv_handle *h, int restart) {
  if (h->impl && h->impl->m >= restart) return DGADV_OK;
  if (h->impl) {   // a longer restart: the basis is reallocated, the old buffers stay with the handle
    cudaStreamSynchronize(h->stream);
    implicit_release(h);
  }
  h->impl = new (std::nothrow) ImplicitState();
  if (!h->impl) return DGADV_ENOMEM;
  const size_t mark = h->allocs.size();
  const int e = allocate_state(h, h->impl, restart);
  if (e != DGADV_OK) {   // none half made: a later call starts over
    implicit_release(h);
    dev_free_from(h, mark);
    cudaGetLastError();
  }
  return e;
}

template <typename T, int P>
int load_tables(dgadv_handle *h) {
  if (h->impl->tablesLoaded) return DGADV_OK;
  const cudaError_t e = upload_itab<T, P>(h->tables, h->stream);
  if (e != cudaSuccess) { h->err = std::string("implicit tables: ") + cudaGetErrorString(e); return DGADV_ECUDA; }
  h->impl->tablesLoaded = true;
  return DGADV_OK;
}

int check_handle(dgadv_handle *h) {
  if (!(h->flags & DGADV_FLAG_IMPLICIT)) {
    h->err = "implicit steps need a handle created with DGADV_FLAG_IMPLICIT";
    return DGADV_EINVAL;
  }
  if (h->prec == DGADV_DF32) { h->err = "implicit steps run in FP64 or FP32"; return DGADV_EUNSUPPORTED; }
  if (!h->hasVelocity) { h->err = "no velocity data"; return DGADV_EINVAL; }
  return DGADV_OK;
}

template <typename T, int P>
int run(dgadv_handle *h, int what, int nSteps, int nStep0, double tau, int ord, double tol, int maxIter,
        int32_t *iters, double *res) {
  if (int e = load_tables<T, P>(h)) return e;
  Solver<T, P> s(h);
  int it = 0;
  double rr = 0.0;
  int e = what == 0 ? s.dirk_steps(nSteps, nStep0, tau, ord, tol, maxIter, it, rr) : s.stationary(tol, maxIter, it, rr);
  if (iters) *iters = it;
  if (res) *res = rr;
  if (e == DGADV_ENOCONV) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "GMRES stopped at relative residual %.3e after %d iterations", rr, it);
    h->err = buf;
  } else if (e == DGADV_ECUDA) {
    h->err = std::string("implicit solve: ") + cudaGetErrorString(cudaGetLastError());
  }
  return e;
}

template <typename T>
int run_t(dgadv_handle *h, int what, int nSteps, int nStep0, double tau, int ord, double tol, int maxIter,
          int32_t *iters, double *res) {
  switch (h->p) {
    case 0: return run<T, 0>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
    case 1: return run<T, 1>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
    case 2: return run<T, 2>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
    case 3: return run<T, 3>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
  }
  return DGADV_EUNSUPPORTED;
}

int dispatch(dgadv_handle *h, int what, int nSteps, int nStep0, double tau, int ord, double tol, int maxIter,
             int restart, int32_t *iters, double *res) {
  if (int e = check_handle(h)) return e;
  if (!(tol > 0.0) || maxIter < 1 || restart < 1 || restart > 256) return DGADV_EINVAL;
  if (int e = ensure_state(h, restart)) return e;
  if (h->prec == DGADV_FP64) return run_t<double>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
  return run_t<float>(h, what, nSteps, nStep0, tau, ord, tol, maxIter, iters, res);
}

}  // namespace
}  // namespace dgadv

using namespace dgadv;

extern "C" int dgadv_step_implicit(dgadv_handle *h, int32_t nSteps, int32_t nStep0, double tau, int32_t ordRK,
                                   const dgadv_krylov *kr, int32_t *iters, double *relres) {
  return guarded(h, [&]() -> int {
  if (!h || nSteps < 0 || !(tau > 0.0) || ordRK < 1 || ordRK > 4) return DGADV_EINVAL;
  DG_CUDA(cudaSetDevice(h->device));
  const dgadv_krylov d = kr ? *kr : dgadv_krylov{1e-12, 2000, 50};
  if (nSteps == 0) return DGADV_OK;
  return dispatch(h, 0, nSteps, nStep0, tau, ordRK, d.tol, d.maxIter, d.restart, iters, relres);
  });
}

extern "C" int dgadv_solve_stationary(dgadv_handle *h, const dgadv_krylov *kr, int32_t *iters, double *relres) {
  return guarded(h, [&]() -> int {
  if (!h) return DGADV_EINVAL;
  DG_CUDA(cudaSetDevice(h->device));
  const dgadv_krylov d = kr ? *kr : dgadv_krylov{1e-12, 2000, 50};
  return dispatch(h, 1, 0, 0, 1.0, 1, d.tol, d.maxIter, d.restart, iters, relres);
  });
}
