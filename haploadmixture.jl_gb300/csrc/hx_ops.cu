// hx_ops.cu -- decode, checks, synthetic data, reductions, EM normalisation,
// projection, batched QP and ZAL quasi-Newton kernels (all FP64 where the
// arithmetic is floating point).
#include "hx_ops.cuh"
#include "hx_qp_dense.cuh"
#include <algorithm>
#include <climits>

namespace hx {

namespace {
constexpr unsigned FULL = 0xffffffffu;

// ------------------------------------------------------------------ decode
// Four bytes (16 individuals) of a SNP row from byte address a on; bytes at or
// past end read as 0.
__device__ __noinline__ uint32_t load_codes(const uint8_t* a, const uint8_t* end) {
    uint32_t v = 0u;
    for (int b = 0; b < 4; ++b)
        if (a + b < end) v |= (uint32_t)a[b] << (8 * b);
    return v;
}

// One round of a 16 x 16 transpose of 2-bit elements: exchanges the blocks off the
// diagonal of each 2H x 2H block (m: the columns of its first half).
template <int H>
__device__ __forceinline__ void swap_round(uint32_t (&x)[16], uint32_t m) {
#pragma unroll
    for (int t = 0; t < 16; ++t)
        if (!(t & H)) {
            const uint32_t a = x[t], b = x[t + H < 16 ? t + H : t];
            x[t] = (a & m) | ((b & m) << (2 * H));
            x[t + H < 16 ? t + H : t] = ((a >> (2 * H)) & m) | (b & ~m);
        }
}

// Decodes word columns jw0 .. jw0+ncol-1 (the 16 SNP rows of word column jw0 + w
// start at bed + 16 w bps) into class words, and counts the blocks whose two SNPs
// are both missing (src/utils.jl:1-18: over all Jf blocks of the file, beyond
// the J that the fit uses).  Thread: 16 individuals x `per` word columns; the 16
// rows' words are transposed as a 16 x 16 matrix of 2-bit codes in registers (four
// rounds of swaps), so the matrix is read once, in words, and each row of 16
// class words is written whole.  Memory-bound.
__global__ void __launch_bounds__(128)
k_pack(const uint8_t* __restrict__ bed, int64_t bps, const uint8_t* end, int64_t I, int64_t J, int64_t Jf, int64_t Ipad,
       int JW, int64_t jw0, int64_t ncol, int per, uint32_t* __restrict__ G, unsigned long long* __restrict__ dm) {
    __shared__ uint4 swap[128 * 4];
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t i0 = 16 * c;              // individuals past Ipad (the last warps) are neither read nor written
    const int nv = (int)min((int64_t)16, max((int64_t)0, I - i0));        // individuals here
    const bool aligned = ((reinterpret_cast<uintptr_t>(bed) | (uintptr_t)bps) & 3u) == 0;
    const uint32_t vmask = nv == 16 ? 0xFFFFFFFFu : (1u << (2 * nv)) - 1u;
    unsigned cnt[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) cnt[r] = 0u;
    const int64_t w1 = min(ncol, ((int64_t)blockIdx.y + 1) * per);
    for (int64_t w = (int64_t)blockIdx.y * per; w < w1; ++w) {
        const int64_t jw = jw0 + w;
        // codes of the 16 rows; rows past the file read as homozygous, individuals
        // past I as missing.  Away from the buffer's end the loads need no checks
        // of their own, so they are all in flight together.
        uint32_t x[16];
        const uint8_t* row = bed + 16 * w * bps + 4 * c;
        if (nv > 0 && 16 * jw + 15 < 2 * Jf && row + 15 * bps + 8 <= end) {
            if (aligned) {
#pragma unroll
                for (int t = 0; t < 16; ++t) x[t] = *reinterpret_cast<const uint32_t*>(row + t * bps);
            } else {
                uint32_t y[16];
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    const uint32_t* p = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(row + t * bps) & ~(uintptr_t)3);
                    x[t] = p[0];
                    y[t] = p[1];
                }
#pragma unroll
                for (int t = 0; t < 16; ++t)
                    x[t] = __funnelshift_r(x[t], y[t], 8 * (unsigned)(reinterpret_cast<uintptr_t>(row + t * bps) & 3u));
            }
        } else {
#pragma unroll
            for (int t = 0; t < 16; ++t)
                x[t] = nv > 0 && 16 * jw + t < 2 * Jf ? load_codes(row + t * bps, end) : 0u;
        }
#pragma unroll
        for (int t = 0; t < 16; ++t) x[t] = (x[t] & vmask) | (0x55555555u & ~vmask);
        swap_round<8>(x, 0x0000FFFFu);
        swap_round<4>(x, 0x00FF00FFu);
        swap_round<2>(x, 0x0F0F0F0Fu);
        swap_round<1>(x, 0x33333333u);
        // x[r]: individual i0 + r, nibble b the class of block 8 jw + b
        const int nb = (int)min((int64_t)8, max((int64_t)0, J - 8 * jw));   // blocks of the fit in this column
        const uint32_t keep = nb == 8 ? 0xFFFFFFFFu : (1u << (4 * nb)) - 1u;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const uint32_t d = x[r] ^ HX_PAD_WORD, e = d | (d >> 1);
            cnt[r] += 8 - __popc((e | (e >> 2)) & 0x11111111u);
            x[r] = (x[r] & keep) | (HX_PAD_WORD & ~keep);
        }
        if (jw < JW) {
            // through shared memory, so that a warp's stores cover whole lines
            uint4* buf = swap + (threadIdx.x & ~31u) * 4;
            const int lane = threadIdx.x & 31;
#pragma unroll
            for (int r = 0; r < 4; ++r)
                buf[4 * lane + (r ^ ((lane >> 1) & 3))] = make_uint4(x[4 * r], x[4 * r + 1], x[4 * r + 2], x[4 * r + 3]);
            __syncwarp();
            uint4* out = reinterpret_cast<uint4*>(G + jw * Ipad + 16 * (c - lane));
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int u = 32 * r + lane;
                if (16 * (c - lane) + 4 * u < Ipad) out[u] = buf[(u & ~3) + ((u & 3) ^ ((u >> 3) & 3))];
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int r = 0; r < 16; ++r)
        if (r < nv && cnt[r]) atomicAdd(dm + i0 + r, (unsigned long long)cnt[r]);
}

// Counts of the 16 classes over n4 x 4 class words, padding included (the caller
// subtracts it).  Four words at a time: each code's positions of the two SNPs as
// bits, the words' bits side by side in one mask, one population count per class.
__global__ void __launch_bounds__(256) k_census(const uint4* __restrict__ G, int64_t n4,
                                                unsigned long long* __restrict__ counts) {
    __shared__ unsigned hist[16];
    if (threadIdx.x < 16) hist[threadIdx.x] = 0u;
    __syncthreads();
    unsigned n[16];
#pragma unroll
    for (int a = 0; a < 16; ++a) n[a] = 0u;
    for (int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x; t < n4; t += (int64_t)gridDim.x * 256) {
        const uint4 v = G[t];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        // bit planes of the nibbles: word q's bit plane p at bits 4 b + q
        uint32_t p[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t x = w[q] & (0x11111111u << b);
                p[b] |= q >= b ? x << (q - b) : x >> (b - q);
            }
        const uint32_t s1[4] = {~p[0] & ~p[1], p[0] & ~p[1], ~p[0] & p[1], p[0] & p[1]};
        const uint32_t s2[4] = {~p[2] & ~p[3], p[2] & ~p[3], ~p[2] & p[3], p[2] & p[3]};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) n[code_g(a) * 4 + code_g(b)] += __popc(s1[a] & s2[b]);
    }
#pragma unroll
    for (int a = 0; a < 16; ++a) {
        const unsigned s = __reduce_add_sync(FULL, n[a]);
        if ((threadIdx.x & 31) == 0) atomicAdd(&hist[a], s);
    }
    __syncthreads();
    if (threadIdx.x < 16 && hist[threadIdx.x]) atomicAdd(counts + threadIdx.x, (unsigned long long)hist[threadIdx.x]);
}

// ------------------------------------------------------------------ synthetic
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t draw53(uint64_t key, uint64_t idx) {
    return mix64(key + (idx + 1) * 0x9E3779B97F4A7C15ULL) >> 11;
}

__global__ void k_synth(uint64_t seed, int64_t I, int64_t J, int K, const uint64_t* __restrict__ thrQ,
                        const uint64_t* __restrict__ thrP, uint64_t thr_miss, uint8_t* __restrict__ bed) {
    const int64_t bps = (I + 3) / 4;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= bps) return;
    const uint64_t k0 = mix64(seed ^ (0ULL * 0x9E3779B97F4A7C15ULL));
    const uint64_t k1 = mix64(seed ^ (1ULL * 0x9E3779B97F4A7C15ULL));
    const uint64_t k2 = mix64(seed ^ (2ULL * 0x9E3779B97F4A7C15ULL));
    for (int64_t j = blockIdx.y; j < J; j += gridDim.y) {
        unsigned o1 = 0, o2 = 0;
        for (int r = 0; r < 4; ++r) {
            const int64_t i = 4 * c + r;
            if (i >= I) break;
            int a1 = 0, a2 = 0;
            for (int cp = 0; cp < 2; ++cp) {
                const uint64_t idx = ((uint64_t)i * (uint64_t)J + (uint64_t)j) * 2 + cp;
                const uint64_t u = draw53(k0, idx);
                int z = K - 1;
                for (int k = 0; k < K; ++k)
                    if (u < thrQ[(int64_t)K * i + k]) { z = k; break; }
                const uint64_t u2 = draw53(k1, idx);
                int h = 3;
                for (int l = 0; l < 4; ++l)
                    if (u2 < thrP[(int64_t)K * (4 * j + l) + z]) { h = l; break; }
                a1 += h >> 1;
                a2 += h & 1;
            }
            unsigned c1 = a1 == 0 ? 0u : (a1 == 1 ? 2u : 3u);
            unsigned c2 = a2 == 0 ? 0u : (a2 == 1 ? 2u : 3u);
            if (draw53(k2, (uint64_t)i * (uint64_t)(2 * J) + (uint64_t)(2 * j)) < thr_miss) c1 = 1u;
            if (draw53(k2, (uint64_t)i * (uint64_t)(2 * J) + (uint64_t)(2 * j + 1)) < thr_miss) c2 = 1u;
            o1 |= c1 << (2 * r);
            o2 |= c2 << (2 * r);
        }
        bed[(2 * j) * bps + c] = (uint8_t)o1;
        bed[(2 * j + 1) * bps + c] = (uint8_t)o2;
    }
}

// ------------------------------------------------------------------ reductions
// Chunk sums [S][NV][ld] (values 0 .. K-1 the gradient, then the Hessian's upper
// triangle) added in chunk order -> Xtz and both triangles of XtX.  Block: 32
// rows; a warp sums one value of 32 consecutive rows (coalesced), and the
// results leave through shared memory, so that the K x K blocks are written in
// order too (each thread walking all values of its own row took 83 us for 5,000
// rows of 20 values and 61 chunks: 20 blocks of uncoalesced stores).
constexpr int RS_ROWS = 32;
__global__ void __launch_bounds__(256) k_reduce_sym(const double* __restrict__ part, int S, int K, int NV, int64_t rows,
                                                    int64_t ld, double* __restrict__ XtX, double* __restrict__ Xtz) {
    extern __shared__ double tile[];   // [NV][RS_ROWS + 1]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t r0 = (int64_t)blockIdx.x * RS_ROWS, r = r0 + lane;
    for (int v = warp; v < NV; v += 8) {
        double s = 0.0;
        if (r < rows) {
            const double* src = part + (int64_t)v * ld + r;
#pragma unroll 8
            for (int c = 0; c < S; ++c) s += src[(int64_t)c * NV * ld];
        }
        tile[v * (RS_ROWS + 1) + lane] = s;
    }
    __syncthreads();
    const int nr = (int)min((int64_t)RS_ROWS, rows - r0);
    for (int t = tid; t < nr * K; t += 256) Xtz[r0 * K + t] = tile[(t % K) * (RS_ROWS + 1) + t / K];
    if (NV == K) return;
    const int KK = K * K;
    for (int t = tid; t < nr * KK; t += 256) {
        const int row = t / KK, e = t - row * KK, a = e / K, b = e - a * K;
        const int lo = min(a, b), hi = max(a, b);
        XtX[r0 * KK + t] = tile[(K + lo * K - lo * (lo - 1) / 2 + hi - lo) * (RS_ROWS + 1) + row];
    }
}

__global__ void k_reduce_sum(const double* __restrict__ part, int64_t n, double* __restrict__ out) {
    __shared__ double red[256];
    double s = 0.0;
    for (int64_t a = threadIdx.x; a < n; a += 256) s += part[a];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// ------------------------------------------------------------------ projection
// OpenADMIXTURE.project_q! contract restated (Chen & Ye 2011): Euclidean
// projection of v onto {x >= eps, sum x = 1}; same operation order as the oracle.
__device__ void project_simplex(double* v, int n, double eps) {
    double y[HX_KMAX > 4 ? HX_KMAX : 4];
    int idx[HX_KMAX > 4 ? HX_KMAX : 4];
    for (int a = 0; a < n; ++a) { y[a] = v[a] - eps; idx[a] = a; }
    for (int a = 1; a < n; ++a) {
        const int t = idx[a];
        int b = a - 1;
        while (b >= 0 && y[idx[b]] < y[t]) { idx[b + 1] = idx[b]; --b; }
        idx[b + 1] = t;
    }
    const double target = 1.0 - n * eps;
    double tsum = 0.0, tmax = 0.0;
    bool found = false;
    for (int a = 0; a < n - 1; ++a) {
        tsum = tsum + y[idx[a]];
        tmax = (tsum - target) / (a + 1);
        if (tmax >= y[idx[a + 1]]) { found = true; break; }
    }
    if (!found) tmax = (tsum + y[idx[n - 1]] - target) / n;
    for (int a = 0; a < n; ++a) {
        const double t = y[a] - tmax;
        v[a] = (t > 0.0 ? t : 0.0) + eps;
    }
}

// src/algorithms_inner.jl:66,75: q_next = project(q .* Xtz ./ 2(J - dm)).
__global__ void k_em_q(const double* __restrict__ q, const double* __restrict__ Xtz,
                       const unsigned long long* __restrict__ dm, int64_t J, int K, int64_t I, double eps,
                       double* __restrict__ qn) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= I) return;
    double v[HX_KMAX];
    const double den = 2.0 * (double)(J - (int64_t)dm[i]);
    for (int k = 0; k < K; ++k) v[k] = (q[(int64_t)K * i + k] * Xtz[(int64_t)K * i + k]) / den;
    project_simplex(v, K, eps);
    for (int k = 0; k < K; ++k) qn[(int64_t)K * i + k] = v[k];
}

// src/algorithms_inner.jl:67-76: p_next = project(normalise(p .* Xtz)) per (k, quartet).
__global__ void k_em_p(const double* __restrict__ p, const double* __restrict__ Xtz, int K, int64_t J, double eps,
                       double* __restrict__ pn) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)K * J) return;
    const int64_t j = t / K;
    const int k = (int)(t % K);
    double v[4];
    for (int h = 0; h < 4; ++h) {
        const int64_t a = (int64_t)K * (4 * j + h) + k;
        v[h] = p[a] * Xtz[a];
    }
    const double s = v[0] + v[1] + v[2] + v[3];
    for (int h = 0; h < 4; ++h) v[h] /= s;
    project_simplex(v, 4, eps);
    for (int h = 0; h < 4; ++h) pn[(int64_t)K * (4 * j + h) + k] = v[h];
}

__global__ void k_step_q(const double* __restrict__ q, const double* __restrict__ d, int K, int64_t ncol, double eps,
                         double* __restrict__ out, double factor) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncol) return;
    double v[HX_KMAX];
    for (int k = 0; k < K; ++k) v[k] = q[(int64_t)K * i + k] + (d ? factor * d[(int64_t)K * i + k] : 0.0);
    project_simplex(v, K, eps);
    for (int k = 0; k < K; ++k) out[(int64_t)K * i + k] = v[k];
}

__global__ void k_step_p(const double* __restrict__ p, const double* __restrict__ d, int K, int64_t J, double eps,
                         double* __restrict__ out, double factor) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)K * J) return;
    const int64_t j = t / K;
    const int k = (int)(t % K);
    double v[4];
    for (int h = 0; h < 4; ++h) {
        const int64_t a = (int64_t)K * (4 * j + h) + k;
        v[h] = p[a] + (d ? factor * d[a] : 0.0);
    }
    project_simplex(v, 4, eps);
    for (int h = 0; h < 4; ++h) out[(int64_t)K * (4 * j + h) + k] = v[h];
}

// ------------------------------------------------------------------ QP
// Equality form of the P step (src/algorithms_inner.jl:307-310); the other
// forms are in hx_qp.cu.
constexpr int QP_WARPS = 4;

__global__ void __launch_bounds__(32 * QP_WARPS)
k_qp_p_eq(int K, int64_t n, const double* __restrict__ XtX, const double* __restrict__ Xtz,
          const double* __restrict__ p, double* __restrict__ pdiff, double* slots) {
    extern __shared__ double smem_qp[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t j = (int64_t)blockIdx.x * QP_WARPS + warp;
    if (j >= n) return;
    const int nv = 4 * K;
    QPWork w = carve(smem_qp + warp * (qp_warp_bytes(nv, K) / sizeof(double)), nv, K);
    for (int a = lane; a < nv; a += 32) {
        const double pa = p[(int64_t)nv * j + a];
        w.d[a] = 0.0;
        w.z[a] = Xtz[(int64_t)nv * j + a];
        w.lo[a] = 0.0 - pa;
        w.hi[a] = 1.0 - pa;
        w.st[a] = (w.lo[a] >= 0.0 && w.hi[a] <= 0.0) ? QL : QF;
        w.d[a] = w.st[a] == QL ? w.lo[a] : 0.0;
    }
    __syncwarp();
    HP H{XtX + (int64_t)K * K * 4 * j, K, 0.0};
    const int it = warp_qp<true>(nv, K, H, w);
    __syncwarp();
    for (int a = lane; a < nv; a += 32) pdiff[(int64_t)nv * j + a] = w.d[a];
    if (it < 0 && lane == 0) atomicAdd(slots + S_QP_FAIL, 1.0);
}

// ------------------------------------------------------------------ ZAL QN
constexpr int QN_THREADS = 256;

// Secant-pair update and the dot products of the QN point: for ZAL UtU (full),
// UtV and Utd with d = x - x_next; for LB (the LBQN step) YtY and Ytd with
// Y = U - V formed per element (a short Y, v close to u, keeps its accuracy).
template <int QS, bool LB>
__global__ void __launch_bounds__(QN_THREADS)
k_qn_dots(int64_t n, const double* __restrict__ x, const double* __restrict__ xn, const double* __restrict__ xn2,
          double* __restrict__ U, double* __restrict__ V, const double* __restrict__ slots, double* __restrict__ part) {
    constexpr int NV = LB ? QS * QS + QS : QS * QS * 2 + QS;
    __shared__ double red[QN_THREADS / 32][NV];
    const int it = (int)slots[S_ITER];
    const int col = (it > 0 ? it - 1 : 0) % QS;
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    for (int64_t a = (int64_t)blockIdx.x * QN_THREADS + threadIdx.x; a < n; a += (int64_t)gridDim.x * QN_THREADS) {
        const double xa = x[a], xna = xn[a];
        const double ua = xna - xa, va = xn2[a] - xna;
        U[a + n * col] = ua;
        V[a + n * col] = va;
        double u[QS], v[QS];
#pragma unroll
        for (int r = 0; r < QS; ++r) {
            u[r] = (r == col) ? ua : U[a + n * r];
            v[r] = (r == col) ? va : V[a + n * r];
        }
        const double dxa = xa - xna;
        if (LB) {
            double y[QS];
#pragma unroll
            for (int r = 0; r < QS; ++r) y[r] = u[r] - v[r];
#pragma unroll
            for (int r = 0; r < QS; ++r) {
#pragma unroll
                for (int s = 0; s < QS; ++s) acc[r * QS + s] += y[r] * y[s];
                acc[QS * QS + r] += y[r] * dxa;
            }
        } else {
#pragma unroll
            for (int r = 0; r < QS; ++r) {
#pragma unroll
                for (int s = 0; s < QS; ++s) {
                    acc[r * QS + s] += u[r] * u[s];
                    acc[QS * QS + r * QS + s] += u[r] * v[s];
                }
                acc[2 * QS * QS + r] += u[r] * dxa;
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double s = acc[v];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[warp][v] = s;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < QN_THREADS / 32; ++w) s += red[w][threadIdx.x];
        part[(int64_t)blockIdx.x * NV + threadIdx.x] = s;
    }
}

// Sums the block partials in block order, then solves (U'U - U'V) c = U'(x - x_next)
// on the first m = min(iter, QS) secant pairs (Gaussian elimination with
// partial pivoting, as Julia's `\`).
// The Q x Q system of the QN point, solved as Julia's `\` (Gaussian
// elimination with partial pivoting): ZAL (lb = 0) (U'U - U'V) c = U'd;
// LBQN (lb = 1) (U-V)'(U-V) c = (U-V)'d.
__global__ void k_qn_solve(const double* __restrict__ part, int nblk, int QS, const double* __restrict__ slots,
                           double* __restrict__ coef, int lb) {
    __shared__ double tot[2 * HX_QMAX_DEV * HX_QMAX_DEV + HX_QMAX_DEV];
    const int NV = lb ? QS * QS + QS : QS * QS * 2 + QS;
    for (int v = threadIdx.x; v < NV; v += blockDim.x) {
        double s = 0.0;
        for (int b = 0; b < nblk; ++b) s += part[(int64_t)b * NV + v];
        tot[v] = s;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    const int it = (int)slots[S_ITER];
    const int m = it < QS ? it : QS;
    double A[HX_QMAX_DEV * HX_QMAX_DEV], b[HX_QMAX_DEV];
    for (int r = 0; r < m; ++r) {
        for (int s = 0; s < m; ++s)
            A[r + m * s] = lb ? tot[r * QS + s] : tot[r * QS + s] - tot[QS * QS + r * QS + s];
        b[r] = lb ? tot[QS * QS + r] : tot[2 * QS * QS + r];
    }
    for (int c = 0; c < m; ++c) {
        int piv = c;
        for (int r = c + 1; r < m; ++r)
            if (fabs(A[r + m * c]) > fabs(A[piv + m * c])) piv = r;
        if (piv != c) {
            for (int k = 0; k < m; ++k) { double t = A[c + m * k]; A[c + m * k] = A[piv + m * k]; A[piv + m * k] = t; }
            double t = b[c]; b[c] = b[piv]; b[piv] = t;
        }
        const double dc = A[c + m * c];
        for (int r = c + 1; r < m; ++r) {
            const double f = A[r + m * c] / dc;
            for (int k = c; k < m; ++k) A[r + m * k] -= f * A[c + m * k];
            b[r] -= f * b[c];
        }
    }
    for (int r = m - 1; r >= 0; --r) {
        double t = b[r];
        for (int k = r + 1; k < m; ++k) t -= A[r + m * k] * b[k];
        b[r] = t / A[r + m * r];
    }
    for (int r = 0; r < QS; ++r) coef[r] = r < m ? b[r] : 0.0;
}

__global__ void k_qn_apply(int64_t n, const double* __restrict__ xn, const double* __restrict__ V, int QS,
                           const double* __restrict__ coef, double* __restrict__ xt) {
    for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
        double t = 0.0;
        for (int r = 0; r < QS; ++r) t += V[a + n * r] * coef[r];
        xt[a] = xn[a] - t;
    }
}

// ------------------------------------------------------------------ bookkeeping
__global__ void k_iter_begin(double* slots) {
    slots[S_ITER] += 1.0;
    slots[S_LL_PREV] = slots[S_LL_NEW];
}

// src/algorithms_outer.jl:154-161: keep the ZAL point only if ll_basic < ll_qn.
__global__ void k_accept(int64_t n, double* __restrict__ x, const double* __restrict__ xt,
                         const double* __restrict__ xn2, double* slots) {
    const double lb = slots[S_LL_BASIC], lq = slots[S_LL_QN];
    const bool qn = lb < lq;
    const double* src = qn ? xt : xn2;
    for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x)
        x[a] = src[a];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const double ll = qn ? lq : lb;
        const double prev = slots[S_LL_PREV];
        slots[S_LL_NEW] = ll;
        slots[S_RELDIFF] = fabs((ll - prev) / prev);
        slots[S_ACCEPT_QN] = qn ? 1.0 : 0.0;
    }
}

__global__ void k_copy_slot(double* slots, int dst, int src) { slots[dst] = slots[src]; }

__global__ void k_nan_check(const double* __restrict__ a, int64_t n, double* slots) {
    bool bad = false;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        bad |= isnan(a[t]);
    if (__any_sync(FULL, bad) && (threadIdx.x & 31) == 0) slots[S_NAN] = 1.0;
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ================================================================== launchers
cudaError_t launch_pack(const uint8_t* bed, int64_t bps, int64_t nbytes, int64_t I, int64_t J, int64_t Jf,
                        int64_t Ipad, int JW, int64_t jw0, int64_t ncol, uint32_t* G, unsigned long long* dm,
                        cudaStream_t st) {
    if (ncol <= 0) return cudaSuccess;
    // word columns per thread: enough CTAs to fill the chip, few additions to dm
    const unsigned gx = nblk(Ipad / 16, 128);
    const int64_t per = std::max<int64_t>(1, std::min<int64_t>(64, ncol * gx / 2432));
    dim3 grid(gx, nblk(ncol, (int)per));
    k_pack<<<grid, 128, 0, st>>>(bed, bps, bed + nbytes, I, J, Jf, Ipad, JW, jw0, ncol, (int)per, G, dm);
    return cudaGetLastError();
}
cudaError_t launch_census(const uint32_t* G, int64_t Ipad, int JW, unsigned long long* counts, cudaStream_t st) {
    const int64_t n4 = Ipad / 4 * JW;
    k_census<<<(unsigned)std::min<int64_t>((n4 + 255) / 256, 1216), 256, 0, st>>>(reinterpret_cast<const uint4*>(G), n4,
                                                                              counts);
    return cudaGetLastError();
}
cudaError_t launch_synth(uint64_t seed, int64_t I, int64_t J, int K, const uint64_t* thrQ, const uint64_t* thrP,
                         double miss, uint8_t* bed, cudaStream_t st) {
    const int64_t bps = (I + 3) / 4;
    const double tm = ceil(miss * 9007199254740992.0);
    const uint64_t thr_miss = tm <= 0.0 ? 0ULL : (uint64_t)tm;
    dim3 grid(nblk(bps, 128), (unsigned)(J < 65535 ? J : 65535));
    k_synth<<<grid, 128, 0, st>>>(seed, I, J, K, thrQ, thrP, thr_miss, bed);
    return cudaGetLastError();
}
cudaError_t launch_reduce_sym(const double* part, int S, int K, bool hess, int64_t rows, int64_t ld, double* XtX,
                              double* Xtz, cudaStream_t st) {
    const int NV = K + (hess ? K * (K + 1) / 2 : 0);
    const size_t smem = (size_t)NV * (RS_ROWS + 1) * sizeof(double);   // <= 23.8 KB (K = 12)
    k_reduce_sym<<<nblk(rows, RS_ROWS), 256, smem, st>>>(part, S, K, NV, rows, ld, XtX, Xtz);
    return cudaGetLastError();
}
cudaError_t launch_reduce_sum(const double* part, int64_t n, double* out, cudaStream_t st) {
    k_reduce_sum<<<1, 256, 0, st>>>(part, n, out);
    return cudaGetLastError();
}
cudaError_t launch_em_q(const double* q, const double* Xtz, const unsigned long long* dm, int64_t J, int K, int64_t I,
                        double eps, double* q_next, cudaStream_t st) {
    k_em_q<<<nblk(I, 128), 128, 0, st>>>(q, Xtz, dm, J, K, I, eps, q_next);
    return cudaGetLastError();
}
cudaError_t launch_em_p(const double* p, const double* Xtz, int K, int64_t J, double eps, double* p_next,
                        cudaStream_t st) {
    k_em_p<<<nblk((int64_t)K * J, 128), 128, 0, st>>>(p, Xtz, K, J, eps, p_next);
    return cudaGetLastError();
}
cudaError_t launch_step_q(const double* q, const double* d, int K, int64_t ncol, double eps, double* out,
                          cudaStream_t st, double factor) {
    k_step_q<<<nblk(ncol, 128), 128, 0, st>>>(q, d, K, ncol, eps, out, factor);
    return cudaGetLastError();
}
cudaError_t launch_step_p(const double* p, const double* d, int K, int64_t J, double eps, double* out,
                          cudaStream_t st, double factor) {
    k_step_p<<<nblk((int64_t)K * J, 128), 128, 0, st>>>(p, d, K, J, eps, out, factor);
    return cudaGetLastError();
}
__global__ void k_f2d(const float* __restrict__ a, int64_t n, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = (double)a[t];
}
cudaError_t launch_f2d(const float* a, int64_t n, double* out, cudaStream_t st) {
    k_f2d<<<nblk(n, 256), 256, 0, st>>>(a, n, out);
    return cudaGetLastError();
}
__global__ void k_d2f(const double* __restrict__ a, int64_t n, float* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = (float)a[t];
}
cudaError_t launch_d2f(const double* a, int64_t n, float* out, cudaStream_t st) {
    k_d2f<<<nblk(n, 256), 256, 0, st>>>(a, n, out);
    return cudaGetLastError();
}
int resident_ctas(const void* kernel, int threads, size_t dyn_smem) {
    cudaFuncAttributes at{};
    int dev = 0, regs_sm = 0, smem_sm = 0, resv = 0, thr_sm = 0, blk_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&at, kernel) != cudaSuccess) return 1;
    cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&resv, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
    cudaDeviceGetAttribute(&blk_sm, cudaDevAttrMaxBlocksPerMultiprocessor, dev);
    const int warps = (threads + 31) / 32;
    int n = std::min(blk_sm, thr_sm / (32 * warps));
    const int rwarp = ((at.numRegs + 7) / 8 * 8 * 32 + 255) / 256 * 256;   // registers of one warp
    if (rwarp > 0) {
        const int wsub = (regs_sm / 4) / rwarp;                               // warps per sub-partition
        n = std::min(n, 4 * wsub / warps);
    }
    const size_t per = at.sharedSizeBytes + dyn_smem + (size_t)resv;
    if (per > 0) n = std::min(n, (int)((size_t)smem_sm / per));
    return std::max(n, 1);
}

cudaError_t init_kernel_attrs(int K) {
    cudaError_t e = cudaFuncSetAttribute(k_qp_p_eq, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(QP_WARPS * qp_warp_bytes(4 * HX_KMAX, HX_KMAX)));
    return e == cudaSuccess ? init_qp_attrs(K) : e;
}
cudaError_t launch_qp_p(int K, int64_t n, int64_t I, const double* XtX, const double* Xtz, const double* p, double rho,
                        double* pdiff, double* slots, int8_t* ws, cudaStream_t st, bool eq) {
    if (!eq) return launch_qp_p_pen(K, n, I, XtX, Xtz, p, rho, pdiff, slots, ws, st);
    const size_t smem = QP_WARPS * qp_warp_bytes(4 * K, K);
    k_qp_p_eq<<<nblk(n, QP_WARPS), 32 * QP_WARPS, smem, st>>>(K, n, XtX, Xtz, p, pdiff, slots);
    return cudaGetLastError();
}
int qn_dots_blocks(int64_t n) {
    int64_t b = (n + QN_THREADS * 8 - 1) / (QN_THREADS * 8);
    return (int)(b < 1 ? 1 : (b > 1216 ? 1216 : b));
}
cudaError_t launch_qn(int64_t n, const double* x, const double* xn, const double* xn2, double* U, double* V, int Qs,
                      double* part, double* coef, double* xt, double* slots, cudaStream_t st, int mode) {
    const int nb = qn_dots_blocks(n);
#define HX_QN(QQ)                                                                                       \
    case QQ:                                                                                            \
        if (mode == 1) k_qn_dots<QQ, true><<<nb, QN_THREADS, 0, st>>>(n, x, xn, xn2, U, V, slots, part);  \
        else k_qn_dots<QQ, false><<<nb, QN_THREADS, 0, st>>>(n, x, xn, xn2, U, V, slots, part);          \
        break;
    switch (Qs) {
        HX_QN(1) HX_QN(2) HX_QN(3) HX_QN(4) HX_QN(5) HX_QN(6)
        default: return cudaErrorInvalidValue;
    }
#undef HX_QN
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_qn_solve<<<1, 128, 0, st>>>(part, nb, Qs, slots, coef, mode == 1 ? 1 : 0);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_qn_apply<<<nblk(n, 256) < 2432 ? nblk(n, 256) : 2432, 256, 0, st>>>(n, xn, V, Qs, coef, xt);
    return cudaGetLastError();
}
cudaError_t launch_iter_begin(double* slots, cudaStream_t st) {
    k_iter_begin<<<1, 1, 0, st>>>(slots);
    return cudaGetLastError();
}
cudaError_t launch_accept(int64_t n, double* x, const double* xt, const double* xn2, double* slots, cudaStream_t st) {
    unsigned nb = nblk(n, 256);
    k_accept<<<nb < 2432 ? nb : 2432, 256, 0, st>>>(n, x, xt, xn2, slots);
    return cudaGetLastError();
}
cudaError_t launch_copy_slot(double* slots, int dst, int src, cudaStream_t st) {
    k_copy_slot<<<1, 1, 0, st>>>(slots, dst, src);
    return cudaGetLastError();
}
cudaError_t launch_nan_check(const double* a, int64_t n, double* slots, cudaStream_t st) {
    unsigned nb = nblk(n, 256);
    k_nan_check<<<nb < 1216 ? nb : 1216, 256, 0, st>>>(a, n, slots);
    return cudaGetLastError();
}

}  // namespace hx
