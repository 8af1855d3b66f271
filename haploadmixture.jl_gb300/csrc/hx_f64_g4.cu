// hx_f64_g4.cu -- plain-method pass instantiations for K = 10.
#include "hx_f64_inst.cuh"

namespace hx {
HX_F64_GROUP(4, HX_F64_CASE(10))
}  // namespace hx
