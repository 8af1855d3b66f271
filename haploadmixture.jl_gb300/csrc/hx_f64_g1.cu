// hx_f64_g1.cu -- plain-method pass instantiations for K = 1, 2, 3, 4, 5.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(1, HX_F64_CASE(1) HX_F64_CASE(2) HX_F64_CASE(3) HX_F64_CASE(4) HX_F64_CASE(5))
}  // namespace hx
