// hx_noalloc.cu -- log-likelihood entry point that allocates no device memory.
//
// Some callers cannot or must not allocate device memory at call time.
// Examples: a host framework that hands out all device memory from its own
// pool (the Julia CUDA.jl or PyTorch caching allocators) and forbids side
// allocations; a latency-critical loop where cudaMalloc/cudaFree would
// synchronise the device.  hx_loglikelihood_noalloc evaluates the
// log-likelihood of src/loops.jl:236-258 directly from caller-owned device
// buffers (raw BED bytes, Q, P, output).  Its only scratch (one partial sum
// per CTA) lives in the file-scope array below, which every GPU that loads
// this library holds until the process exits.
#include "hx_ops.cuh"
#include "../../include/haplo_gb300.h"

#include <algorithm>

namespace hx {
namespace {

constexpr int NA_THREADS = 128;
constexpr int NA_STAGE = 16;        // blocks whose p a CTA stages at a time

// Scratch of the no-allocation entry point: one FP64 partial per CTA.
__device__ __align__(256) double g_noalloc_scratch[HX_NOALLOC_SCRATCH];

// One pair again in FP64, its mantissa and exponent folded in separately.
template <int K>
__device__ __noinline__ void redo_f64(unsigned nib, const double* qr, const double* pj, float& mant, int& ex, bool& zero,
                                      bool& bad) {
    double qd[4], Ld, ud[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < K; ++k) s = fma(qr[k], pj[h * K + k], s);
        qd[h] = s;
    }
    pair_eval<double>(nib, qd, Ld, ud);
    if (!(Ld > 0.0)) {
        if (Ld == 0.0) zero = true; else bad = true;
        return;
    }
    mant = renorm(mant * (float)renorm(Ld, ex), ex);
}

// Mixed method (the plain FP64 one is k_loglik64 in hx_pass_f64.cu): one
// individual per thread over a chunk of blocks, decoding the two SNP codes
// of each block straight from the BED bytes (src/loops.jl:55-71); pair
// likelihoods multiply into an exponent-renormalised product (one log per
// CTA).  The CTA converts p to FP32 once per stage: a conversion is an FP64
// operation, 64 clocks of a quarter of an SM for a warp, and with 4 K of them per
// pair the kernel did little else (20,000 individuals x 10,000 blocks, K = 8:
// 11.2 -> 0.90 ms).  Writes one partial per CTA into scratch[blockIdx.y * gridDim.x + blockIdx.x].
template <int K>
__global__ void __launch_bounds__(NA_THREADS)
k_loglik_bed(const uint8_t* __restrict__ bed, int64_t bps, int64_t I, int64_t J, const double* __restrict__ q,
             const double* __restrict__ p, int64_t per_chunk, double* __restrict__ scratch) {
    __shared__ float sp[NA_STAGE * 4 * K];
    __shared__ double red[NA_THREADS / 32];
    __shared__ long long rex[NA_THREADS / 32];
    const int tid = threadIdx.x;
    const int64_t i = (int64_t)blockIdx.x * NA_THREADS + tid;
    const bool active = i < I;
    const int64_t j0 = (int64_t)blockIdx.y * per_chunk;
    const int64_t j1 = min(J, j0 + per_chunk);
    float qi[K];
#pragma unroll
    for (int k = 0; k < K; ++k) qi[k] = active ? (float)q[(int64_t)K * i + k] : 1.f / K;
    float mant = 1.f;
    int ex = 0;
    bool zero = false, bad = false;
    const int64_t byte = active ? i >> 2 : 0;
    const int sh = 2 * (int)(i & 3);
    for (int64_t js = j0; js < j1; js += NA_STAGE) {
        const int nb = (int)min((int64_t)NA_STAGE, j1 - js);
        unsigned codes[NA_STAGE];               // both codes of each block of the stage
#pragma unroll
        for (int b = 0; b < NA_STAGE; ++b) {
            codes[b] = NIB_MM;
            if (active && b < nb) {
                const uint8_t* r = bed + 2 * (js + b) * bps + byte;
                codes[b] = ((r[0] >> sh) & 3u) | (((r[bps] >> sh) & 3u) << 2);
            }
        }
        __syncthreads();
        for (int t = tid; t < nb * 4 * K; t += NA_THREADS) sp[t] = (float)p[(int64_t)K * 4 * js + t];
        __syncthreads();
#pragma unroll
        for (int b = 0; b < NA_STAGE; ++b) {
            const unsigned nib = codes[b];
            if (nib == NIB_MM) continue;
            const float* pj = sp + 4 * K * b;
            float qp[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                float s = 0.f;
#pragma unroll
                for (int k = 0; k < K; ++k) s = fma(qi[k], pj[h * K + k], s);
                qp[h] = s;
            }
            float L, u[4];
            pair_eval<float>(nib, qp, L, u);
            if (L < 1.17549435e-38f && L == L) {
                // FP32 pair likelihood below the smallest normal float (caller
                // Q/P entries far below the fit's 1e-5 floor): the renormaliser
                // reads the exponent field, so redo this pair in FP64 and fold
                // its mantissa and exponent in separately
                redo_f64<K>(nib, q + (int64_t)K * i, p + (int64_t)K * 4 * (js + b), mant, ex, zero, bad);
                continue;
            }
            if (!(L > 0.f)) {
                if (L == 0.f) zero = true; else bad = true;
                L = 1.f;
            }
            mant = renorm(mant * L, ex);
        }
    }
    // the CTA's product, exponents apart, and one log
    double m = mant;
    long long e = ex;
    auto mul = [&](double y) {
        int x = 0;
        m = renorm(m * y, x);
        e += x;
    };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, m, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
        mul(y);
    }
    const bool any_zero = __syncthreads_or(zero), any_bad = __syncthreads_or(bad);
    if ((tid & 31) == 0) { red[tid >> 5] = m; rex[tid >> 5] = e; }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < NA_THREADS / 32; ++w) { e += rex[w]; mul(red[w]); }
        double v = log(m) + (double)e * 0.69314718055994530942;
        if (any_zero) v = -INFINITY;
        if (any_bad) v = NAN;
        scratch[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = v;
    }
}

// Sums the n partials in a fixed order into *out (one CTA).
__global__ void k_sum_partials(const double* __restrict__ scratch, int64_t n, double* __restrict__ out) {
    __shared__ double red[256];
    double s = 0.0;
    for (int64_t a = threadIdx.x; a < n; a += 256) s += scratch[a];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

#define HX_NA_FOR_K(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

cudaError_t launch_bed(int K, dim3 grid, cudaStream_t st, const uint8_t* bed, int64_t bps, int64_t I, int64_t J,
                       const double* q, const double* p, int64_t per_chunk, double* scratch) {
#define HX_CASE(KK) \
    case KK: k_loglik_bed<KK><<<grid, NA_THREADS, 0, st>>>(bed, bps, I, J, q, p, per_chunk, scratch); break;
    switch (K) { HX_NA_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
    return cudaGetLastError();
}

}  // namespace
}  // namespace hx

extern "C" int hx_loglikelihood_noalloc(const uint8_t* d_bed, int64_t bytes_per_snp, int64_t I, int64_t J, int32_t K,
                                        const double* d_q, const double* d_p, int32_t precision, double* d_ll,
                                        void* stream) {
    using namespace hx;
    if (!d_bed || !d_q || !d_p || !d_ll || I <= 0 || J <= 0 || bytes_per_snp < (I + 3) / 4) return HX_EINVAL;
    if (K < 1 || K > HX_KMAX) return HX_EUNSUPPORTED;
    if (precision != HX_PREC_FP64 && precision != HX_PREC_MIXED) return HX_EINVAL;
    // one partial per CTA: (individual tiles) x (block chunks) must fit the static scratch
    const int64_t tiles = (I + NA_THREADS - 1) / NA_THREADS;
    if (tiles > HX_NOALLOC_SCRATCH) return HX_EUNSUPPORTED;
    // The device address of the scratch array in the current device's
    // context (host code may not use the symbol itself as an address).  It is
    // looked up on every call, not cached: after a device or primary-context
    // reset the module is loaded again at another address.  The lookup
    // allocates nothing; the first call in a context also loads the module,
    // so make that first call before any stream capture.
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) return HX_ECUDA;
    double* scratch = (double*)ptr;
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == HX_PREC_FP64) {
        // chunks of whole word columns (8 blocks), as many CTAs as run at once
        const int64_t JW = (J + 7) / 8;
        int64_t S = std::max<int64_t>(1, std::min<int64_t>(JW, (1216 + tiles - 1) / tiles));
        S = std::min<int64_t>(S, HX_NOALLOC_SCRATCH / tiles);
        const int64_t per = (JW + S - 1) / S;
        S = (JW + per - 1) / per;
        PassArgs a{};
        a.I = I; a.J = J; a.JW = (int)JW;
        a.q = d_q; a.p = d_p; a.S = (int)S; a.per_chunk = (int)per; a.part = scratch;
        if (launch_loglik_f64_bed(K, a, d_bed, bytes_per_snp, st) != cudaSuccess) return HX_ECUDA;
        k_sum_partials<<<1, 256, 0, st>>>(scratch, tiles * S, d_ll);
        return cudaGetLastError() == cudaSuccess ? HX_OK : HX_ECUDA;
    }
    const int64_t target = 2048;
    int64_t S = std::max<int64_t>(1, std::min<int64_t>(J, (target + tiles - 1) / tiles));
    S = std::min<int64_t>(S, HX_NOALLOC_SCRATCH / tiles);
    const int64_t per_chunk = (J + S - 1) / S;
    S = (J + per_chunk - 1) / per_chunk;
    dim3 grid((unsigned)tiles, (unsigned)S);
    if (launch_bed(K, grid, st, d_bed, bytes_per_snp, I, J, d_q, d_p, per_chunk, scratch) != cudaSuccess)
        return HX_ECUDA;
    k_sum_partials<<<1, 256, 0, st>>>(scratch, tiles * S, d_ll);
    if (cudaGetLastError() != cudaSuccess) return HX_ECUDA;
    return HX_OK;
}
