// The transport problem on the device (transport/*.m, configuration 'rotation' without coupling
// to a shallow-water model): several species on one mesh, each advected as its depth-integrated
// concentration c h with the depth-integrated velocity, only over its active elements, with the
// linear vertex limiter applied to its concentration c.
//
// Per Runge-Kutta stage, for all species at once (transport/solveSubStep.m; dgadv_transport.cuh):
//   k_tr_stage   c h <- SSP update with the masked advective term of c;  c <- Pi(c h / h)
//   k_tr_limit   c <- linear vertex limiter, zero Dirichlet data;  c h <- Pi(c h)
// and at the step's last stage the species' masks follow from that limiter call's patch
// extremes (transport/postprocessStep.m, core/computeMask.m).  The handle supplies the mesh,
// the depth-integrated velocity (dgadv_set_velocity) and the limiter; each species has its own
// vertex keys and global extremes.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "dgadv_handle.h"

namespace dgadv {

struct TransportState {
  int nSpecies = 0, capacity = 0;   // species in use, species the buffers hold
  double maskTol = 1e-6;
  bool isMask = true;
  // all species one after the other; cHs: c h between the stages of a step
  void *cH = nullptr, *cHs = nullptr, *conc = nullptr, *work = nullptr;
  uint8_t *mask = nullptr;
  void *hQ = nullptr;               // depth at the volume points, Q x Kp
  void *vkeys = nullptr;
  unsigned long long *slots = nullptr;
  long long pass = 0;               // limiter passes so far (which key set)
};

void transport_release(dgadv_handle *h) {
  delete h->trans;   // device buffers belong to h->allocs
  h->trans = nullptr;
}

}  // namespace dgadv

using namespace dgadv;

namespace {

double rk_table_transport(int ord, double omega[3], double cst[3]) {
  omega[0] = omega[1] = omega[2] = 0.0;
  cst[0] = 0.0; cst[1] = 1.0; cst[2] = 0.5;   // core/rungeKuttaExplicit.m:64-78
  if (ord == 2) { omega[1] = 0.5; return 2; }
  if (ord == 3) { omega[1] = 0.75; omega[2] = 1.0 / 3.0; return 3; }
  return 1;
}

int check(dgadv_handle *h) {
  if (!h->trans) { h->err = "dgadv_transport_init was not called"; return DGADV_EINVAL; }
  return DGADV_OK;
}

TrArgs species_args(const dgadv_handle *h) {
  const TransportState *st = h->trans;
  TrArgs a{};
  a.nSpecies = st->nSpecies;
  a.conc = st->conc; a.work = st->work; a.mask = st->mask; a.hQ = st->hQ;
  a.cHin = st->cH; a.cH0 = st->cH; a.cHout = st->cH;
  a.vkeys = st->vkeys; a.slots = st->slots;
  a.maskTol = st->maskTol;
  return a;
}
// Both kernels of a stage (or of the initial data), and the next pass's key sets.
int stage_of_all(dgadv_handle *h, TrArgs &a, double tBC) {
  TransportState *st = h->trans;
  const PrecOps &o = ops_of(h);
  a.pass = st->pass;
  for (int m = 0; m < h->nTerms; ++m) a.gco[m] = h->timeFn[m] == DGADV_TIME_EXP_NEG ? std::exp(-tBC) : 1.0;
  DG_CUDA(o.tr_stage(h, a));
  DG_CUDA(o.tr_limit(h, a));
  ++st->pass;
  return DGADV_OK;
}

}  // namespace

extern "C" int dgadv_transport_init(dgadv_handle *h, int32_t nSpecies, const double *hDisc, const double *cH0,
                                    double maskTol, int32_t isMask) {
  return guarded(h, [&]() -> int {
  if (!h || nSpecies < 1 || nSpecies > 64 || !hDisc || !cH0 || !(maskTol >= 0.0)) return DGADV_EINVAL;
  const PrecOps &o = ops_of(h);
  if (!o.tr_stage) { h->err = "the transport kernels are built for FP32 and FP64"; return DGADV_EUNSUPPORTED; }
  if (!h->lim || h->limType != DGADV_LIM_LINEAR || h->p < 1 || (h->flags & DGADV_FLAG_IMPLICIT)) {
    h->err = "transport needs an explicit handle with the linear limiter and p >= 1";
    return DGADV_EINVAL;
  }
  if (!h->hasVelocity) { h->err = "dgadv_set_velocity was not called"; return DGADV_EINVAL; }
  DG_CUDA(cudaSetDevice(h->device));
  const size_t K = h->K, Kp = h->Kp, N = h->N, Q = h->Q;
  const size_t bytes = N * Kp * o.realBytes;
  const size_t nKeys = (size_t)2 * h->Vp, nSlots = (size_t)h->nInst * kSlotCopies * 2;
  int e;
  // buffers kept from an earlier call that hold as many species; the handle frees them
  if (h->trans && h->trans->capacity < nSpecies) transport_release(h);
  if (!h->trans) {
    TransportState *n = new (std::nothrow) TransportState();
    if (!n) return DGADV_ENOMEM;
    h->trans = n;
    const size_t mark = h->allocs.size();
    if ((e = dev_alloc(h, &n->cH, nSpecies * bytes)) || (e = dev_alloc(h, &n->cHs, nSpecies * bytes)) ||
        (e = dev_alloc(h, &n->conc, nSpecies * bytes)) || (e = dev_alloc(h, &n->work, nSpecies * bytes)) ||
        (e = dev_alloc(h, (void **)&n->mask, nSpecies * Kp)) || (e = dev_alloc(h, &n->hQ, Q * Kp * o.realBytes)) ||
        (e = dev_alloc(h, &n->vkeys, 3 * nSpecies * nKeys * o.keyBytes)) ||
        (e = dev_alloc(h, (void **)&n->slots, 3 * nSpecies * nSlots * 8))) {
      transport_release(h);
      dev_free_from(h, mark);
      cudaGetLastError();
      return e;
    }
    n->capacity = nSpecies;
  }
  TransportState *st = h->trans;
  st->nSpecies = nSpecies;
  st->maskTol = maskTol;
  st->isMask = isMask != 0;
  st->pass = 0;
  // depth at the volume points (internal element order)
  std::vector<double> hq(Q * Kp, 1.0);
  for (size_t k = 0; k < K; ++k) {
    const int ext = h->permv[k];
    for (size_t q = 0; q < Q; ++q) {
      double v = 0.0;
      for (size_t j = 0; j < N; ++j) v += h->tables.phiQ[q * N + j] * hDisc[j * K + ext];
      hq[q * Kp + k] = v;
    }
  }
  if ((e = upload_real(h, st->hQ, hq))) return e;
  DG_CUDA(cudaMemsetAsync(st->cH, 0, nSpecies * bytes, h->stream));
  DG_CUDA(cudaMemsetAsync(st->cHs, 0, nSpecies * bytes, h->stream));
  DG_CUDA(cudaMemsetAsync(st->conc, 0, nSpecies * bytes, h->stream));
  DG_CUDA(cudaMemsetAsync(st->work, 0, nSpecies * bytes, h->stream));
  DG_CUDA(cudaMemsetAsync(st->mask, 1, nSpecies * Kp, h->stream));
  // every key set reset: each species' minima at the largest key, maxima at 0
  for (size_t i = 0; i < (size_t)3 * nSpecies; ++i) {
    unsigned char *v = (unsigned char *)st->vkeys + i * nKeys * o.keyBytes;
    DG_CUDA(cudaMemsetAsync(v, 0xFF, (size_t)h->Vp * o.keyBytes, h->stream));
    DG_CUDA(cudaMemsetAsync(v + (size_t)h->Vp * o.keyBytes, 0, (size_t)h->Vp * o.keyBytes, h->stream));
  }
  std::vector<unsigned long long> slots(3 * nSpecies * nSlots);
  for (size_t i = 0; i < slots.size(); ++i) slots[i] = (i & 1) ? 0ULL : o.slotKeyMax;
  if ((e = upload(h, st->slots, slots.data(), slots.size() * 8))) return e;
  DG_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // the uploads have landed
  for (int s = 0; s < nSpecies; ++s) {
    DG_CUDA(cudaMemcpyAsync(h->stage_ext, cH0 + (size_t)s * K * N, K * N * sizeof(double), cudaMemcpyHostToDevice,
                            h->stream));
    DG_CUDA(o.scatter_in(h, (unsigned char *)st->cH + s * bytes));
  }
  // transport/initializeProblem.m: c = Pi(c h / h), limited at t = 0, c h = Pi(c h), mask
  TrArgs a = species_args(h);
  a.init = true;
  a.updateMask = st->isMask;
  if ((e = stage_of_all(h, a, 0.0))) return e;
  DG_CUDA(cudaStreamSynchronize(h->stream));
  return dgadv_sync(h);
  });
}

extern "C" int dgadv_transport_step(dgadv_handle *h, int32_t nSteps, int32_t nStep0, double tau) {
  return guarded(h, [&]() -> int {
  if (!h || nSteps < 0 || !(tau > 0.0)) return DGADV_EINVAL;
  if (int e = check(h)) return e;
  DG_CUDA(cudaSetDevice(h->device));
  TransportState *st = h->trans;
  double omega[3], cst[3];
  const int S = (int)rk_table_transport(h->ordRK, omega, cst);
  for (int n = 0; n < nSteps; ++n) {
    const double t0 = (double)(nStep0 + n) * tau;
    for (int i = 0; i < S; ++i) {
      // boundary time of the limiter (transport/solveSubStep.m): the next stage's time
      const double tBC = (i + 1 < S) ? t0 + cst[i + 1] * tau : t0 + tau;
      TrArgs a = species_args(h);
      a.cHin = i == 0 ? st->cH : st->cHs;
      a.cHout = i == S - 1 ? st->cH : st->cHs;   // c h of the step's start is read no more by then
      a.omega = omega[i]; a.tau = tau;
      a.updateMask = i == S - 1 && st->isMask;
      if (int e = stage_of_all(h, a, tBC)) return e;
    }
  }
  return dgadv_sync(h);
  });
}

extern "C" int dgadv_transport_get(dgadv_handle *h, int32_t species, double *cH, double *conc, uint8_t *mask) {
  return guarded(h, [&]() -> int {
  if (!h) return DGADV_EINVAL;
  if (int e = check(h)) return e;
  TransportState *st = h->trans;
  if (species < 0 || species >= st->nSpecies) return DGADV_EINVAL;
  DG_CUDA(cudaSetDevice(h->device));
  const PrecOps &o = ops_of(h);
  const size_t KN = (size_t)h->K * h->N, bytes = (size_t)h->N * h->Kp * o.realBytes;
  if (cH) {
    DG_CUDA(o.gather_out(h, (unsigned char *)st->cH + species * bytes));
    DG_CUDA(cudaMemcpyAsync(cH, h->stage_ext, KN * 8, cudaMemcpyDeviceToHost, h->stream));
    DG_CUDA(cudaStreamSynchronize(h->stream));
  }
  if (conc) {
    DG_CUDA(o.gather_out(h, (unsigned char *)st->conc + species * bytes));
    DG_CUDA(cudaMemcpyAsync(conc, h->stage_ext, KN * 8, cudaMemcpyDeviceToHost, h->stream));
    DG_CUDA(cudaStreamSynchronize(h->stream));
  }
  if (mask) {
    std::vector<uint8_t> m(h->K);
    DG_CUDA(cudaMemcpyAsync(m.data(), st->mask + (size_t)species * h->Kp, h->K, cudaMemcpyDeviceToHost, h->stream));
    DG_CUDA(cudaStreamSynchronize(h->stream));
    for (int k = 0; k < h->K; ++k) mask[h->permv[k]] = m[k];
  }
  return dgadv_sync(h);
  });
}
