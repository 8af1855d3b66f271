// hx_accum_f64_g2.cu -- general passes of the plain method, K = 9 .. 12.
#include "hx_accum_f64.cuh"

namespace hx {
HX_A64_GROUP(2, HX_A64_CASE(9) HX_A64_CASE(10) HX_A64_CASE(11) HX_A64_CASE(12))
}  // namespace hx
