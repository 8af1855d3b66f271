// hx_f64_g5.cu -- plain-method pass instantiations for K = 11.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(5, HX_F64_CASE(11))
}  // namespace hx
