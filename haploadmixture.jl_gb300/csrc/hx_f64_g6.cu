// hx_f64_g6.cu -- plain-method pass instantiations for K = 12.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(6, HX_F64_CASE(12))
}  // namespace hx
