// hx_f64_g2.cu -- plain-method pass instantiations for K = 6, 7.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(2, HX_F64_CASE(6) HX_F64_CASE(7))
}  // namespace hx
