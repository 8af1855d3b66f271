// hx_accum_f64.cuh -- launches of the plain method's general passes for the K of one
// unit (hx_accum_f64_g*.cu, which compile in parallel).
#pragma once
#include "hx_ops.cuh"

#define HX_A64_CASE(KK)                                                                              \
    case KK:                                                                                         \
        if (p_side) hess ? k_accum_p<KK, double, true><<<grid, ACC_THREADS, 0, st>>>(a, r)           \
                         : k_accum_p<KK, double, false><<<grid, ACC_THREADS, 0, st>>>(a, r);         \
        else hess ? k_accum_q<KK, double, true><<<grid, ACC_THREADS, 0, st>>>(a, r)                  \
                  : k_accum_q<KK, double, false><<<grid, ACC_THREADS, 0, st>>>(a, r);                \
        break;
#define HX_A64_GROUP(g, cases)                                                                       \
    cudaError_t accum_f64_g##g(int K, bool p_side, bool hess, const PassArgs& a, const RunIf& r,     \
                               cudaStream_t st) {                                                    \
        dim3 grid((unsigned)(p_side ? (a.J + 31) / 32 : a.Ipad / ACC_THREADS), (unsigned)a.S);       \
        switch (K) { cases default: return cudaErrorInvalidValue; }                                  \
        return cudaGetLastError();                                                                   \
    }
