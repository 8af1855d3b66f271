// hx_f64_inst.cuh -- launches of the plain-method passes for one K, included by
// the hx_f64_g*.cu units, each of which instantiates a few values of K so that
// they compile in parallel.
#pragma once
#include <algorithm>
#include "hx_f64.cuh"

namespace hx {
namespace {

template <int K, bool HESS, bool PS>
cudaError_t f64_attr() {
    return cudaFuncSetAttribute(k_f64_pass<K, HESS, PS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)f_smem<K, HESS, PS>());
}
template <int K>
cudaError_t f64_attrs_k() {
    cudaError_t e = f64_attr<K, true, false>();
    if (e == cudaSuccess) e = f64_attr<K, true, true>();
    if (e == cudaSuccess) e = f64_attr<K, false, false>();
    if (e == cudaSuccess) e = f64_attr<K, false, true>();
    return e;
}

template <int K, bool HESS, bool PS>
cudaError_t f64_launch(const F64Call& c) {
    using D = FDim<K, HESS>;
    static_assert(f_smem<K, HESS, PS>() <= 232448, "shared memory of one CTA");
    static_assert(D::COLS <= D::TCOLS && D::PER <= D::STR, "TMEM columns");
    const PassArgs& a = c.a;
    const double* v = PS ? a.q : a.p;             // the vectors along the reduction
    const int64_t n = PS ? a.I : 4 * a.J;
    const int64_t stages = PS ? (a.I + F_KD - 1) / F_KD : a.JW;
    const int64_t tiles = PS ? (a.J + 31) / 32 : a.Ipad / 128;
    const int64_t nq = a.I * K, np = 4 * a.J * K;
    const int noff = (int)std::min<int64_t>(F_MAXB, (nq + np + 1023) / 1024);
    k_f64_range<<<noff, 256, 0, c.st>>>(a.q, nq, a.p, np, HESS ? F_LO_HESS : F_LO_GRAD, c.off, c.rare.flag);
    k_f64_img<K, HESS><<<(unsigned)((stages + 3) / 4), 128, 0, c.st>>>(v, n, stages, PS, a.img);
    F64Args fa{stages, c.off, noff, c.rare};
    dim3 grid((unsigned)tiles, (unsigned)a.S, D::NG);
    k_f64_pass<K, HESS, PS><<<grid, F_THREADS, f_smem<K, HESS, PS>(), c.st>>>(a, fa);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    PassArgs g = a;
    g.S = c.Sg;
    g.per_chunk = c.per_chunk_g;
    const RunIf r{c.off, noff};
    e = PS ? launch_accum_p_f64(K, HESS, g, r, c.st) : launch_accum_q_f64(K, HESS, g, r, c.st);
    if (e != cudaSuccess) return e;
    const int64_t rows = PS ? 4 * a.J : a.I;
    return launch_f64_reduce(a.part, a.S, c.Sg, K, HESS, PS && HESS, rows, PS ? rows : a.Ipad, PS ? a.p : a.q, c.off, noff, c.rare,
                             a.XtX, a.Xtz, c.st);
}
template <int K>
cudaError_t f64_launch_k(const F64Call& c) {
    if (c.p_side) return c.hess ? f64_launch<K, true, true>(c) : f64_launch<K, false, true>(c);
    return c.hess ? f64_launch<K, true, false>(c) : f64_launch<K, false, false>(c);
}

}  // namespace
}  // namespace hx

// c == null: set the kernels' attributes
#define HX_F64_CASE(KK) case KK: return c ? f64_launch_k<KK>(*c) : f64_attrs_k<KK>();
#define HX_F64_GROUP(g, cases)                                \
    cudaError_t f64_run_g##g(int K, const F64Call* c) {       \
        switch (K) { cases }                                  \
        return cudaErrorInvalidValue;                         \
    }
