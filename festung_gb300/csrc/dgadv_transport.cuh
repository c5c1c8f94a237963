// Kernels of the transport problem (transport/solveSubStep.m, configuration 'rotation' without
// coupling): species advected as depth-integrated concentrations c h, each only over its active
// elements (its mask).
//
// A stage is two kernels over all species (blockIdx.y), with programmatic dependent launch between
// them; what was a chain of seven small launches per species and stage ran at launch latency.
//
// k_tr_stage: the SSP update of c h from the masked advective term of the concentration c with
//   the depth-integrated velocity (the handle's velocity factors), then the new concentration
//   c = Pi(c h / h), unlimited, and its mean to the species' vertex keys.  An inactive element keeps
//   its c h.  An active element's outflow counts across an edge to an active element or a
//   boundary edge, its inflow only from an active neighbour (the masked branches of
//   core/assembleMatElemDphiPhiFuncDiscVec.m:115-141 and core/assembleMatEdgePhiPhiValUpwind.m).
//   The reference's transport keeps hatM = I (transport/preprocessProblem.m), so the mass solve
//   is the division by detJ already folded into the factors.
// k_tr_limit: the linear vertex limiter, c h = Pi(c h), and after the last stage the mask
//   (core/computeMask.m, 'vertex-based'): an element is active if at one of its vertices
//   the patch maximum minus the patch minimum of the element means (with the reference's global
//   shift and the zero Dirichlet data of the limiter call) reaches the tolerance.
// Projections use point values at the volume rule with hatM = I (core/projectDataQ0T2DataDisc.m).
//
// Both run 64 elements per block: the reference's mesh has 8192, and FP64 instructions issue
// once in 19 cycles per SM, so a few species have to spread over every SM.  8192 triangles, p = 1,
// four species, one step (two stages): 282 -> 50 us; 524288 triangles 2432 -> 1917 us.
#pragma once
#include "dgadv_launch.cuh"

namespace dgadv {

constexpr int kTrBlock = 64;

struct VolWeights {
  double w[12];
};

// s = Pi(a / h) (TOCONC) or Pi(a h); h: the depth at the element's volume points, stride Kp.
template <typename T, int P, bool TOCONC>
__device__ __forceinline__ void tr_convert(const T *a, const T *h, size_t Kp, const VolWeights &wq, T *s) {
  constexpr int N = Dims<P>::N, Q = Dims<P>::Q;
  const Tab<T, P> &tb = tab<T, P>();
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = T(0);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    T v = T(0);
#pragma unroll
    for (int j = 0; j < N; ++j) v = fma(tb.phiQ[q][j], a[j], v);
    const T hq = h[(size_t)q * Kp];
    v = TOCONC ? v / hq : v * hq;
    const T wv = T(wq.w[q]) * v;
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = fma(wv, tb.phiQ[q][i], s[i]);
  }
}

template <typename T> struct TrDev {
  const T *conc, *cHin, *cH0;
  T *work;
  const uint8_t *mask;     // written by k_tr_limit of the step before: not __restrict__
  const T *hQ;
  LimOut<T> lo;            // species 0's; species s at s times the strides
  size_t keyStride, slotStride;
  double omega, tau;
  int init;
};

template <typename T, int P>
__global__ void __launch_bounds__(kTrBlock) k_tr_stage(const Geo<T> g, const TrDev<T> a, const VolWeights wq) {
  constexpr int N = Dims<P>::N, Q = Dims<P>::Q, R = Dims<P>::R;
  const int k = blockIdx.x * kTrBlock + threadIdx.x, s = blockIdx.y;
  const Tab<T, P> &tb = tab<T, P>();
  const size_t Kp = g.Kp, at = (size_t)s * N * Kp;
  const T *conc = a.conc + at, *cHin = a.cHin + at, *cH0 = a.cH0 + at;
  const uint8_t *mask = a.mask + (size_t)s * Kp;
  LimOut<T> lo = a.lo;
  lo.vkeys += s * a.keyStride; lo.vreset += s * a.keyStride;
  lo.slots += s * a.slotStride; lo.reset += s * a.slotStride;
  const bool active = k < g.K;
  int vid[3] = {0, 0, 0};
  if (active) { vid[0] = g.V0T[k]; vid[1] = g.V0T[Kp + k]; vid[2] = g.V0T[2 * Kp + k]; }
  pdl_wait();
  pdl_trigger();
  reset_next<T>(g, lo, k);
  T q0 = T(0);
  if (active) {
    T cdot[N], cH[N], c1[N];
#pragma unroll
    for (int i = 0; i < N; ++i) cdot[i] = T(0);
    if (!a.init && mask[k]) {
      T c[N];
#pragma unroll
      for (int i = 0; i < N; ++i) c[i] = conc[i * Kp + k];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        T cq = T(0);
#pragma unroll
        for (int j = 0; j < N; ++j) cq = fma(tb.phiQ[q][j], c[j], cq);
        const T f1 = g.F[q * Kp + k] * cq, f2 = g.F[(Q + q) * Kp + k] * cq;
#pragma unroll
        for (int i = 0; i < N; ++i) cdot[i] = fma(tb.g2[q][i], f2, fma(tb.g1[q][i], f1, cdot[i]));
      }
      const int code = g.code[k];
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        const int nb = g.nbr[n * Kp + k];
        const int np = (code >> (2 * n)) & 3;
        const bool outOk = (code >> (6 + n)) & 1;
        const bool act = nb >= 0 && mask[nb];
        const bool outCounts = nb >= 0 ? act : outOk;
        T cn[N];
#pragma unroll
        for (int j = 0; j < N; ++j) cn[j] = act ? conc[j * Kp + nb] : T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T v = g.Vn[(n * R + r) * Kp + k];
          T tr = T(0);
          if (v > T(0) && outCounts) {
#pragma unroll
            for (int j = 0; j < N; ++j) tr = fma(tb.phi1D[n][r][j], c[j], tr);
          } else if (v < T(0) && act) {
            for (int j = 0; j < N; ++j) tr = fma(tb.thetaPhi[n][np & 3][r][j], cn[j], tr);
          }
          const T fl = v * tr;
#pragma unroll
          for (int i = 0; i < N; ++i) cdot[i] = fma(-tb.phi1D[n][r][i], fl, cdot[i]);
        }
      }
    }
    if (a.init) {
#pragma unroll
      for (int i = 0; i < N; ++i) cH[i] = cHin[i * Kp + k];
    } else {
      const T w = T(a.omega), tt = T(a.tau);
#pragma unroll
      for (int i = 0; i < N; ++i) cH[i] = w * cH0[i * Kp + k] + (T(1) - w) * (cHin[i * Kp + k] + tt * cdot[i]);
    }
    tr_convert<T, P, true>(cH, a.hQ + k, Kp, wq, c1);
#pragma unroll
    for (int i = 0; i < N; ++i) a.work[at + i * Kp + k] = c1[i];
    q0 = lin_mean<T, P>(c1);
  }
  scatter_quantities<T, 1>(g, lo, &q0, vid, active);
}

template <typename T, int P>
__global__ void __launch_bounds__(kTrBlock) k_tr_limit(const Geo<T> g, const T *work, T *conc, T *cH, uint8_t *mask,
                                                       const T *hQ, LimIn<T> li, size_t keyStride, size_t slotStride,
                                                       double tol, int updateMask, const StageScalars sc,
                                                       const VolWeights wq) {
  constexpr int N = Dims<P>::N;
  __shared__ T sh[2];
  const int k = blockIdx.x * kTrBlock + threadIdx.x, s = blockIdx.y;
  const size_t Kp = g.Kp, at = (size_t)s * N * Kp;
  li.vkeys += s * keyStride;
  li.slots += s * slotStride;
  const bool active = k < g.K;
  int vid[3] = {0, 0, 0}, dmask = 0;
  T data[3] = {T(0), T(0), T(0)};
  if (active) {
    vid[0] = g.V0T[k]; vid[1] = g.V0T[Kp + k]; vid[2] = g.V0T[2 * Kp + k];
    dmask = (g.code[k] >> 9) & 7;
    if (g.cDV0T)
      for (int m = 0; m < g.nTerms; ++m) {
        const T gm = T(sc.gco[m]);
#pragma unroll
        for (int n = 0; n < 3; ++n) data[n] += gm * g.cDV0T[((size_t)m * 3 + n) * Kp + k];
      }
  }
  pdl_wait();
  pdl_trigger();
  if (li.shift) load_shifts<T>(li.slots + slot_base(g, 1), 1, sh);
  T c[N];
#pragma unroll
  for (int i = 0; i < N; ++i) c[i] = active ? work[at + i * Kp + k] : T(0);
  VKeys<T, 1> kv;
  load_vkeys<T, 1>(g, li, vid, kv);
  __syncthreads();
  if (!active) return;
  limit_lin_element<T, P, false>(li, kv, sh, dmask, data, c);   // these kernels are bound by latency: plain FP64
  bool bad = false;
#pragma unroll
  for (int i = 0; i < N; ++i) { conc[at + i * Kp + k] = c[i]; bad |= !finite_(c[i]); }
  if (bad) atomicOr(sc.flag, 1);
  T out[N];
  tr_convert<T, P, false>(c, hQ + k, Kp, wq, out);
#pragma unroll
  for (int i = 0; i < N; ++i) cH[at + i * Kp + k] = out[i];
  if (updateMask) {
    T valD[3], mn[3], mx[3];
#pragma unroll
    for (int n = 0; n < 3; ++n) valD[n] = ((dmask >> n) & 1) ? T(0) : T(NAN);
    patch_minmax<T, 1>(li, kv, sh, 0, valD, mn, mx);
    const T d = fmax(fmax(mx[0] - mn[0], mx[1] - mn[1]), mx[2] - mn[2]);
    mask[(size_t)s * Kp + k] = d >= T(tol) ? 1 : 0;
  }
}

// The species' key sets of a pass (three sets rotate, as the handle's own: lim_out).
template <typename T> struct TrKeys {
  typename KeyOf<T>::type *vkeys, *vreset;
  unsigned long long *slots, *reset;
  size_t keyStride, slotStride;
};
template <typename T> static TrKeys<T> tr_keys(const dgadv_handle *h, const TrArgs &a) {
  using K_ = typename KeyOf<T>::type;
  TrKeys<T> r;
  const int set = (int)(a.pass % 3), next = (set + 1) % 3;
  r.keyStride = (size_t)2 * h->Vp;
  r.slotStride = (size_t)h->nInst * kSlotCopies * 2;
  r.vkeys = (K_ *)a.vkeys + set * a.nSpecies * r.keyStride;
  r.vreset = (K_ *)a.vkeys + next * a.nSpecies * r.keyStride;
  r.slots = a.slots + set * a.nSpecies * r.slotStride;
  r.reset = a.slots + next * a.nSpecies * r.slotStride;
  return r;
}
template <int P> static VolWeights tr_weights(const dgadv_handle *h) {
  VolWeights wq{};
  for (int q = 0; q < Dims<P>::Q && q < 12; ++q) wq.w[q] = h->tables.vol.W[q];
  return wq;
}
// Launch over (blocks, species) on the handle's stream with programmatic dependent launch.
template <typename... KArgs, typename... Args>
static void launch_tr(const dgadv_handle *h, void (*kern)(KArgs...), int grid, int nSpecies, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, nSpecies);
  cfg.blockDim = dim3(kTrBlock);
  cfg.stream = h->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (h->flags & DGADV_FLAG_NO_PDL) ? 0 : 1;
  cudaLaunchKernelEx(&cfg, kern, args...);
}

template <typename T, int P>
static cudaError_t launch_tr_stage(dgadv_handle *h, const TrArgs &a) {
  const TrKeys<T> kk = tr_keys<T>(h, a);
  TrDev<T> d{};
  d.conc = (const T *)a.conc; d.cHin = (const T *)a.cHin; d.cH0 = (const T *)a.cH0; d.work = (T *)a.work;
  d.mask = a.mask; d.hQ = (const T *)a.hQ;
  d.lo.vkeys = kk.vkeys; d.lo.vreset = kk.vreset; d.lo.slots = kk.slots; d.lo.reset = kk.reset;
  d.lo.nc = 1; d.lo.type = 0;
  d.keyStride = kk.keyStride; d.slotStride = kk.slotStride;
  d.omega = a.omega; d.tau = a.tau; d.init = a.init ? 1 : 0;
  const int grid = (std::max(h->K, h->numV) + kTrBlock - 1) / kTrBlock;   // blocks also reset vertex keys
  launch_tr(h, k_tr_stage<T, P>, grid, a.nSpecies, make_geo<T>(h), d, tr_weights<P>(h));
  return cudaGetLastError();
}
template <typename T, int P>
static cudaError_t launch_tr_limit(dgadv_handle *h, const TrArgs &a) {
  const TrKeys<T> kk = tr_keys<T>(h, a);
  LimIn<T> li{};
  li.vkeys = kk.vkeys; li.slots = kk.slots; li.nc = 1; li.type = 0;
  li.shift = (h->flags & DGADV_FLAG_NO_SHIFT) ? 0 : 1;
  StageScalars sc{};
  sc.flag = h->flag;
  for (int m = 0; m < 4; ++m) sc.gco[m] = a.gco[m];
  launch_tr(h, k_tr_limit<T, P>, (h->K + kTrBlock - 1) / kTrBlock, a.nSpecies, make_geo<T>(h), (const T *)a.work,
            (T *)a.conc, (T *)a.cHout, a.mask, (const T *)a.hQ, li, kk.keyStride, kk.slotStride, a.maskTol,
            a.updateMask ? 1 : 0, sc, tr_weights<P>(h));
  return cudaGetLastError();
}

template <typename T, int MASK>
static cudaError_t dispatch_tr_stage(dgadv_handle *h, const TrArgs &a) {
  switch (h->p) {
    case 1: if constexpr ((MASK & 2) != 0) return launch_tr_stage<T, 1>(h, a); break;
    case 2: if constexpr ((MASK & 4) != 0) return launch_tr_stage<T, 2>(h, a); break;
    case 3: if constexpr ((MASK & 8) != 0) return launch_tr_stage<T, 3>(h, a); break;
  }
  return cudaErrorNotSupported;
}
template <typename T, int MASK>
static cudaError_t dispatch_tr_limit(dgadv_handle *h, const TrArgs &a) {
  switch (h->p) {
    case 1: if constexpr ((MASK & 2) != 0) return launch_tr_limit<T, 1>(h, a); break;
    case 2: if constexpr ((MASK & 4) != 0) return launch_tr_limit<T, 2>(h, a); break;
    case 3: if constexpr ((MASK & 8) != 0) return launch_tr_limit<T, 3>(h, a); break;
  }
  return cudaErrorNotSupported;
}

// The operation table of a unit with the transport kernels added.
template <typename T, int MASK>
static PrecOps with_transport(PrecOps o) {
  o.tr_stage = dispatch_tr_stage<T, MASK>;
  o.tr_limit = dispatch_tr_limit<T, MASK>;
  return o;
}

}  // namespace dgadv
