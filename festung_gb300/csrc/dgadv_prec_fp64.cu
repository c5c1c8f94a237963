// Kernels and launch sequences of the FP64 path (stored reals: double), every degree, with the adjoint
// and transport kernels.  The persistent and the linked step, whose kernels hold the stage kernels'
// code once more, compile beside it (dgadv_prec_fp64_multi.cu).
#include "dgadv_device.cuh"

namespace dgadv {
DGADV_DEFINE_TABLES(double, cTd)
DGADV_DEFINE_DIGIT_TABLES(cFx)
}  // namespace dgadv

#include "dgadv_launch.cuh"
#include "dgadv_adjoint.cuh"
#include "dgadv_transport.cuh"

namespace dgadv {
const PrecOps &ops_fp64() {
  static const PrecOps ops = add_fp64_multi(with_transport<double, 0xF>(with_adjoint<double, 0xF>(make_ops<double, 0xF, true>())));
  return ops;
}
}  // namespace dgadv
