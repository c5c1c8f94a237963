// The FP64 persistent step and linked step (every degree), with their own copy of the constant tables.
#include "dgadv_device.cuh"

namespace dgadv {
DGADV_DEFINE_TABLES(double, cTd)
DGADV_DEFINE_DIGIT_TABLES(cFx)
}  // namespace dgadv

#include "dgadv_launch.cuh"
#include "dgadv_persist.cuh"
#include "dgadv_linked.cuh"

namespace dgadv {
PrecOps add_fp64_multi(PrecOps o) {
  o = with_linked<double>(with_persistent<double, 0xF>(o));
  o.upload_tables_more = upload_tables_p<double, 0xF>;
  return o;
}
}  // namespace dgadv
