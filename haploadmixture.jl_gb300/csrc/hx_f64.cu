// hx_f64.cu -- dispatch of the plain (FP64) method's passes on K, and the
// reduction of their chunk sums.
#include "hx_ops.cuh"
#include <algorithm>

namespace hx {

cudaError_t f64_run_g1(int K, const F64Call* c);   // K = 1..5
cudaError_t f64_run_g2(int K, const F64Call* c);   // K = 6, 7
cudaError_t f64_run_g3(int K, const F64Call* c);   // K = 8, 9
cudaError_t f64_run_g4(int K, const F64Call* c);   // K = 10
cudaError_t f64_run_g5(int K, const F64Call* c);   // K = 11
cudaError_t f64_run_g6(int K, const F64Call* c);   // K = 12

namespace {
cudaError_t f64_run(int K, const F64Call* c) {
    if (K <= 5) return f64_run_g1(K, c);
    if (K <= 7) return f64_run_g2(K, c);
    if (K <= 9) return f64_run_g3(K, c);
    return K == 10 ? f64_run_g4(K, c) : K == 11 ? f64_run_g5(K, c) : f64_run_g6(K, c);
}
}  // namespace

cudaError_t launch_f64_pass(int K, const F64Call& c) { return f64_run(K, &c); }
cudaError_t f64_attrs(int K) { return f64_run(K, nullptr); }

// Bytes of the larger side's stage images (FDim::IMG of the Hessian form, the
// larger one).
size_t f64_image_bytes(int K, int64_t I, int64_t J) {
    const int nv = K * (K + 1) / 2, ng = f64_groups(nv), nhp = f64_nhp((nv + ng - 1) / ng);
    const size_t img = (size_t)ng * F_NDB * nhp * 64 + (size_t)32 * ((K + 1) | 1) * 8;
    return img * (size_t)std::max((J + 7) / 8, (I + 31) / 32);
}

namespace {
// Chunk sums -> XtX (both triangles) and Xtz.  Those of the digit passes (S chunks of
// NH = NV - K values) give Xtz = XtX x (see hx_f64.cuh), or are Xtz itself for the
// gradient-only pass; where the general passes ran (Sg chunks), Xtz leads each chunk.
// Block: 32 rows; a warp sums one value of 32 consecutive rows (coalesced), the results
// go out through shared memory, so that the K x K blocks are written in order too.
constexpr int FR_ROWS = 32;
__global__ void __launch_bounds__(256) k_f64_reduce(const double* __restrict__ part, int S, int Sg, int K, bool hess,
                                                    bool g, int64_t rows, int64_t ld, const double* __restrict__ x,
                                                    const unsigned* __restrict__ off, int noff, F64Rare rare,
                                                    double* __restrict__ XtX, double* __restrict__ Xtz) {
    extern __shared__ double tile[];   // [K + NH][FR_ROWS + 1]: Xtz, then the triangle
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __shared__ int mx[FR_ROWS];            // high word of the row's largest entry of x
    if (tid < FR_ROWS) mx[tid] = 0;
    const bool general = __syncthreads_or(tid < noff && off[tid] != 0u);
    const int NH = hess ? K * (K + 1) / 2 : 0;
    const int64_t r0 = (int64_t)blockIdx.x * FR_ROWS, r = r0 + lane;
    if (general) {
        for (int v = warp; v < K + NH; v += 8) {
            double s = 0.0;
            if (r < rows) {
                const double* src = part + (int64_t)v * ld + r;
#pragma unroll 8
                for (int c = 0; c < Sg; ++c) s += src[(int64_t)c * (K + NH) * ld];
            }
            tile[v * (FR_ROWS + 1) + lane] = s;
        }
    } else {
        const int NV = hess ? NH : K;
        const int flag = *rare.flag;
        int sh = 0;                        // the row's exponent
        if (g) {
            for (int t = tid; t < FR_ROWS * K; t += 256)
                if (r0 * K + t < rows * K) atomicMax(&mx[t / K], __double2hiint(x[r0 * K + t]));
            __syncthreads();
            if (r < rows) sh = -f64_exponent(mx[lane]);
        }
        for (int v = warp; v < NV; v += 8) {
            double s = 0.0;
            if (r < rows) {
                const double* src = part + (int64_t)v * ld + r;
#pragma unroll 8
                for (int c = 0; c < S; ++c) s += src[(int64_t)c * NV * ld];
                if (flag) {                // products of out-of-range weights; left zero for the next pass
                    long long* i = rare.i + (int64_t)v * rows + r;
                    const int64_t word = NV * rows;
                    const long long i0 = i[0], i1 = i[word], i2 = i[2 * word];
                    if (i0 | i1 | i2) {
                        s += scalbn((double)i0, 2) + (scalbn((double)i1, -35) + scalbn((double)i2, -72));
                        i[0] = i[word] = i[2 * word] = 0;
                    }
                }
                s = scalbn(s, sh);
            }
            tile[((hess ? K : 0) + v) * (FR_ROWS + 1) + lane] = s;
        }
        if (hess) {
            __syncthreads();
            for (int t = tid; t < FR_ROWS * K; t += 256) {
                const int row = t / K, a = t - row * K;
                double g = 0.0;
                if (r0 + row < rows)
                    for (int b = 0; b < K; ++b) {
                        const int lo = min(a, b), hi = max(a, b);
                        g = fma(tile[(K + lo * K - lo * (lo - 1) / 2 + hi - lo) * (FR_ROWS + 1) + row],
                                x[(r0 + row) * K + b], g);
                    }
                tile[a * (FR_ROWS + 1) + row] = g;
            }
        }
    }
    __syncthreads();
    const int nr = (int)min((int64_t)FR_ROWS, rows - r0);
    for (int t = tid; t < nr * K; t += 256) Xtz[r0 * K + t] = tile[(t % K) * (FR_ROWS + 1) + t / K];
    if (!hess) return;
    const int KK = K * K;
    for (int t = tid; t < nr * KK; t += 256) {
        const int row = t / KK, e = t - row * KK, a = e / K, b = e - a * K;
        const int lo = min(a, b), hi = max(a, b);
        XtX[r0 * KK + t] = tile[(K + lo * K - lo * (lo - 1) / 2 + hi - lo) * (FR_ROWS + 1) + row];
    }
}
}  // namespace

cudaError_t launch_f64_reduce(const double* part, int S, int Sg, int K, bool hess, bool g, int64_t rows, int64_t ld,
                              const double* x, const unsigned* off, int noff, const F64Rare& rare, double* XtX,
                              double* Xtz, cudaStream_t st) {
    const int NV = K + (hess ? K * (K + 1) / 2 : 0);
    const size_t smem = (size_t)NV * (FR_ROWS + 1) * sizeof(double);   // <= 23.8 KB (K = 12)
    k_f64_reduce<<<(unsigned)((rows + FR_ROWS - 1) / FR_ROWS), 256, smem, st>>>(part, S, Sg, K, hess, g, rows, ld, x,
                                                                                off, noff, rare, XtX, Xtz);
    return cudaGetLastError();
}

}  // namespace hx
