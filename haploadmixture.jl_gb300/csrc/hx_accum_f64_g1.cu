// hx_accum_f64_g1.cu -- general passes of the plain method, K = 1 .. 8, and their dispatch.
#include "hx_accum_f64.cuh"

namespace hx {
HX_A64_GROUP(1, HX_A64_CASE(1) HX_A64_CASE(2) HX_A64_CASE(3) HX_A64_CASE(4) HX_A64_CASE(5) HX_A64_CASE(6)
                HX_A64_CASE(7) HX_A64_CASE(8))
// K = 9 .. 12
cudaError_t accum_f64_g2(int K, bool p_side, bool hess, const PassArgs& a, const RunIf& r, cudaStream_t st);

cudaError_t launch_accum_q_f64(int K, bool hess, const PassArgs& a, const RunIf& r, cudaStream_t st) {
    return K <= 8 ? accum_f64_g1(K, false, hess, a, r, st) : accum_f64_g2(K, false, hess, a, r, st);
}
cudaError_t launch_accum_p_f64(int K, bool hess, const PassArgs& a, const RunIf& r, cudaStream_t st) {
    return K <= 8 ? accum_f64_g1(K, true, hess, a, r, st) : accum_f64_g2(K, true, hess, a, r, st);
}
}  // namespace hx
