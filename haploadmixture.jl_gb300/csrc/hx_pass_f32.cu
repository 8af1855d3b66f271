// hx_pass_f32.cu -- CUDA-core accumulation passes of the mixed method.
#include "hx_ops.cuh"

#define HX_FOR_K(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

namespace hx {

cudaError_t launch_accum_q_f32(int K, bool hess, const PassArgs& a, cudaStream_t st) {
    dim3 grid((unsigned)(a.Ipad / ACC_THREADS), (unsigned)a.S);
#define HX_CASE(KK) \
    case KK: if (hess) k_accum_q<KK, float, true><<<grid, ACC_THREADS, 0, st>>>(a, RunIf{}); \
             else k_grad_q<KK><<<grid, ACC_THREADS, 0, st>>>(a); break;
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
    return cudaGetLastError();
}

cudaError_t launch_accum_p_f32(int K, bool hess, const PassArgs& a, cudaStream_t st) {
    dim3 grid((unsigned)((a.J + 31) / 32), (unsigned)a.S);
#define HX_CASE(KK) \
    case KK: if (hess) k_accum_p<KK, float, true><<<grid, ACC_THREADS, 0, st>>>(a, RunIf{}); \
             else k_accum_p<KK, float, false><<<grid, ACC_THREADS, 0, st>>>(a, RunIf{}); break;
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
    return cudaGetLastError();
}

}  // namespace hx
