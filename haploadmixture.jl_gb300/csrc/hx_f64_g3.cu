// hx_f64_g3.cu -- plain-method pass instantiations for K = 8, 9.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(3, HX_F64_CASE(8) HX_F64_CASE(9))
}  // namespace hx
