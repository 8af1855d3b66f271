// hx_skfr.cu -- AIM selection by sparse k-means with feature ranking (SKFR).
//
// The reference optionally selects ancestry-informative markers before the fit
// (src/driver.jl:60-73, 84-105): SparseKmeansFeatureRanking.sparsekmeans1 on an
// ImputedSnpMatrix with blocks of 2 SNPs, then SnpArrays.filter to the sorted
// AIMs.  That package is not part of the reference tree; this is the published
// method (Zhang, Lange and Xu 2020, SKFR1) on the GPU:
//   features   x = (g - mean) / sd per SNP over observed genotypes (n-1 sd),
//              missing -> 0; a SNP with < 2 observations or no variance -> 0;
//   start      k-means++ over all SNPs, uniform draws from SplitMix64(seed + t);
//   iteration  cluster means (an empty cluster keeps its centre), SNP score
//              sum_j n_j theta_jl^2, the `sparsity` best blocks of 2 SNPs kept
//              (higher score first, lower index on ties), centres zero elsewhere,
//              reassignment to the nearest centre over the kept SNPs (lower
//              cluster index on ties), until no assignment changes or max_iter.
// A SNP's standardised value depends only on its 2-bit code, so features are a
// 4-entry table per SNP read through the packed bytes, and cluster sums are
// integer code counts times that table.  All FP64 arithmetic uses explicit
// round-to-nearest operations in a fixed order (no contraction), so results do
// not depend on the thread schedule.
#include "hx_ops.cuh"
#include "../../include/haplo_gb300.h"

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

namespace hx {
namespace {

constexpr int SK_THREADS = 256;
constexpr int SK_WARPS = SK_THREADS / 32;
constexpr int SK_STAGE = 128;       // SNPs staged per step of the distance pass
constexpr int SK_LOADERS = 128;     // threads that stage them

__device__ __forceinline__ unsigned sk_code(const uint8_t* __restrict__ bed, int64_t bps, int64_t l, int64_t i) {
    return (bed[l * bps + (i >> 2)] >> (2 * (int)(i & 3))) & 3u;
}

// Word w of SNP row l: the codes of individuals 16w .. 16w+15, two bits each.
// Rows start at any byte, so it is cut from two aligned words (the buffer is
// padded past its end); codes past the row's individuals are left to the caller.
__device__ __forceinline__ unsigned sk_word(const uint8_t* __restrict__ bed, int64_t bps, int64_t l, int64_t w) {
    const int64_t o = l * bps + 4 * w;
    const unsigned* p = reinterpret_cast<const unsigned*>(bed + (o & ~(int64_t)3));
    return __funnelshift_r(p[0], p[1], 8 * (int)(o & 3));
}

// Bit 2r of masks[j * W + w]: individual 16w + r is in cluster j (K = 1 without
// assign: every individual).
__global__ void k_sk_masks(const int* __restrict__ assign, int64_t I, int64_t W, int K, unsigned* __restrict__ masks) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= W * K) return;
    const int64_t w = t % W;
    const int j = (int)(t / W);
    unsigned m = 0u;
    for (int r = 0; r < 16; ++r)
        if (16 * w + r < I && (!assign || assign[16 * w + r] == j)) m |= 1u << (2 * r);
    masks[t] = m;
}

// Per SNP (one warp each): counts of the four codes over the first I
// individuals, then (lane 0) the standardised value of each code.
__global__ void __launch_bounds__(SK_THREADS)
k_sk_tables(const uint8_t* __restrict__ bed, int64_t bps, int64_t W, int64_t M, const unsigned* __restrict__ all,
            double* __restrict__ T) {
    const int lane = threadIdx.x & 31;
    const int64_t l = (int64_t)blockIdx.x * SK_WARPS + (threadIdx.x >> 5);
    if (l >= M) return;
    unsigned n[4] = {0u, 0u, 0u, 0u};
    for (int64_t w = lane; w < W; w += 32) {
        const unsigned x = sk_word(bed, bps, l, w), y = x >> 1, m = all[w];
        n[0] += __popc(m & ~x & ~y);
        n[2] += __popc(m & ~x & y);
        n[3] += __popc(m & x & y);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) n[c] = __reduce_add_sync(0xffffffffu, n[c]);
    if (lane != 0) return;
    double t0 = 0.0, t2 = 0.0, t3 = 0.0;
    const double n0 = (double)n[0], n1 = (double)n[2], n2 = (double)n[3];
    const double nobs = __dadd_rn(__dadd_rn(n0, n1), n2);
    if (nobs >= 2.0) {
        const double mu = __ddiv_rn(__dadd_rn(__dmul_rn(n1, 1.0), __dmul_rn(n2, 2.0)), nobs);
        const double a = __dsub_rn(1.0, mu), b = __dsub_rn(2.0, mu);
        const double ss = __dadd_rn(__dadd_rn(__dmul_rn(n0, __dmul_rn(mu, mu)), __dmul_rn(n1, __dmul_rn(a, a))),
                                    __dmul_rn(n2, __dmul_rn(b, b)));
        const double var = __ddiv_rn(ss, __dsub_rn(nobs, 1.0));
        if (var > 0.0) {
            const double sd = __dsqrt_rn(var);
            t0 = __ddiv_rn(__dsub_rn(0.0, mu), sd);
            t2 = __ddiv_rn(a, sd);
            t3 = __ddiv_rn(b, sd);
        }
    }
    T[4 * l + 0] = t0;
    T[4 * l + 1] = 0.0;   // missing: the mean
    T[4 * l + 2] = t2;
    T[4 * l + 3] = t3;
}

// Column t of the centres (theta[l*K + t]) = individual c's features.
__global__ void k_sk_row(const uint8_t* __restrict__ bed, int64_t bps, int64_t c, const double* __restrict__ T,
                         int64_t M, int K, int t, double* __restrict__ theta) {
    for (int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; l < M; l += (int64_t)gridDim.x * blockDim.x)
        theta[l * K + t] = T[4 * l + sk_code(bed, bps, l, c)];
}

// Squared distance terms D2[(s * KK + j) * 4 + c] = (T[l, c] - theta[l, col0 + j])^2
// of SNP l = sel[s], code c and centre j (row stride ldt of theta).
__global__ void k_sk_terms(const double* __restrict__ T, const double* __restrict__ theta, int ldt, int col0, int KK,
                           const int64_t* __restrict__ sel, int64_t nsel, double* __restrict__ D2) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nsel * KK * 4;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = t / (4 * KK), l = sel[s];
        const int j = (int)(t / 4 % KK);
        const double d = __dsub_rn(T[4 * l + t % 4], theta[l * ldt + col0 + j]);
        D2[t] = __dmul_rn(d, d);
    }
}

// Squared distances of 32 individuals per CTA to KK centres, warp j the
// distances to centre j: each is the sum of nsel terms in order, one FP64
// addition per term (the terms come from the table: a SNP's distance to a
// centre has only four values).  The chain of additions is what bounds it, so
// a warp carries one chain per lane and the centres go to different warps.
// With d_out (KK = 1 only) the distance is written there; otherwise the nearest
// centre (lower index on ties) goes to assign and, with dmin, its distance.
// I = 4,000, 20,000 SNPs: 11.2 ms with one thread per individual walking bytes.
// Four more warps stage the next SNPs' terms and codes meanwhile (with the
// summing warps loading for themselves a step took 300 clocks per SNP).
__global__ void __launch_bounds__(32 * HX_KMAX + SK_LOADERS)
k_sk_dist(const uint8_t* __restrict__ bed, int64_t bps, int64_t I, const double* __restrict__ D2, int KK,
          const int64_t* __restrict__ sel, int64_t nsel, int* __restrict__ assign, double* __restrict__ d_out,
          double* __restrict__ dmin) {
    extern __shared__ __align__(16) double sk_sm[];      // [2][SK_STAGE][KK][4] terms, [KK][32] results
    __shared__ uint64_t codes[2][SK_STAGE];              // 8 bytes: 32 individuals
    const int tid = threadIdx.x, j = tid >> 5, lane = tid & 31;
    const int64_t i0 = (int64_t)blockIdx.x * 32, w0 = i0 >> 4;
    double* res = sk_sm + 2 * SK_STAGE * KK * 4;
    auto stage = [&](int buf, int64_t s0) {
        const int n = (int)min((int64_t)SK_STAGE, nsel - s0), t0 = tid - 32 * KK;
        if (t0 < n) {
            const int64_t l = sel[s0 + t0];
            codes[buf][t0] = sk_word(bed, bps, l, w0) | ((uint64_t)sk_word(bed, bps, l, w0 + 1) << 32);
        }
        const double2* src = reinterpret_cast<const double2*>(D2 + s0 * KK * 4);
        double2* dst = reinterpret_cast<double2*>(sk_sm + buf * SK_STAGE * KK * 4);
#pragma unroll 4
        for (int t = t0; t < n * KK * 2; t += SK_LOADERS) dst[t] = src[t];
    };
    double acc = 0.0;
    if (j >= KK && nsel > 0) stage(0, 0);
    for (int64_t s0 = 0, buf = 0; s0 < nsel; s0 += SK_STAGE, buf ^= 1) {
        __syncthreads();
        if (j >= KK) {
            if (s0 + SK_STAGE < nsel) stage((int)buf ^ 1, s0 + SK_STAGE);
            continue;
        }
        const double* t = sk_sm + buf * SK_STAGE * KK * 4 + j * 4;
        const int n = (int)min((int64_t)SK_STAGE, nsel - s0);
        if (n == SK_STAGE) {
#pragma unroll 16
            for (int s = 0; s < SK_STAGE; ++s) acc = __dadd_rn(acc, t[s * KK * 4 + ((codes[buf][s] >> (2 * lane)) & 3u)]);
        } else {
            for (int s = 0; s < n; ++s) acc = __dadd_rn(acc, t[s * KK * 4 + ((codes[buf][s] >> (2 * lane)) & 3u)]);
        }
    }
    if (j < KK) res[j * 32 + lane] = acc;
    __syncthreads();
    const int64_t i = i0 + lane;
    if (j != 0 || i >= I) return;
    if (d_out) {
        d_out[i] = acc;
        return;
    }
    int best = 0;
    for (int c = 1; c < KK; ++c)
        if (res[c * 32 + lane] < res[best * 32 + lane]) best = c;
    assign[i] = best;
    if (dmin) dmin[i] = res[best * 32 + lane];
}

// Per SNP (one warp each): counts of codes 0, 2, 3 per cluster, then the
// cluster means (clusters with n_j = 0 keep their centre) and the SNP's score
// sum_j n_j theta_jl^2.
__global__ void __launch_bounds__(SK_THREADS)
k_sk_centers(const uint8_t* __restrict__ bed, int64_t bps, int64_t W, int64_t M, int K,
             const unsigned* __restrict__ masks, const double* __restrict__ n, const double* __restrict__ T,
             double* __restrict__ theta, double* __restrict__ score) {
    __shared__ unsigned cnt[SK_WARPS][HX_KMAX][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t l = (int64_t)blockIdx.x * SK_WARPS + w;
    if (l < M) {
        // 16 individuals per word: code and membership bits, counted together
        unsigned c[HX_KMAX][3];
#pragma unroll
        for (int j = 0; j < HX_KMAX; ++j) c[j][0] = c[j][1] = c[j][2] = 0u;
        for (int64_t x = lane; x < W; x += 32) {
            const unsigned v = sk_word(bed, bps, l, x), y = v >> 1;
            const unsigned a = ~v & ~y, b = ~v & y, d = v & y;
#pragma unroll
            for (int j = 0; j < HX_KMAX; ++j)
                if (j < K) {
                    const unsigned m = masks[j * W + x];
                    c[j][0] += __popc(m & a);
                    c[j][1] += __popc(m & b);
                    c[j][2] += __popc(m & d);
                }
        }
#pragma unroll
        for (int j = 0; j < HX_KMAX; ++j)
            if (j < K)
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const unsigned t = __reduce_add_sync(0xffffffffu, c[j][e]);
                    if (lane == 0) cnt[w][j][e] = t;
                }
    }
    __syncwarp();
    if (l >= M || lane != 0) return;
    const double t0 = T[4 * l + 0], t2 = T[4 * l + 2], t3 = T[4 * l + 3];
    double sc = 0.0;
    for (int j = 0; j < K; ++j) {
        if (n[j] > 0.0) {
            const double s = __dadd_rn(__dadd_rn(__dmul_rn((double)cnt[w][j][0], t0), __dmul_rn((double)cnt[w][j][1], t2)),
                                       __dmul_rn((double)cnt[w][j][2], t3));
            theta[l * K + j] = __ddiv_rn(s, n[j]);
        }
        const double th = theta[l * K + j];
        sc = __dadd_rn(sc, __dmul_rn(n[j], __dmul_rn(th, th)));
    }
    score[l] = sc;
}

// Centres are zero off the kept SNPs (keep[l] == 0).
__global__ void k_sk_mask(double* __restrict__ theta, const uint8_t* __restrict__ keep, int64_t M, int K) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < M * K; e += (int64_t)gridDim.x * blockDim.x)
        if (!keep[e / K]) theta[e] = 0.0;
}

// D2: scratch of nsel * K * 4 doubles
cudaError_t launch_dist(int K, int64_t I, const uint8_t* bed, int64_t bps, const double* T, const double* theta,
                        int ldt, int col0, const int64_t* sel, int64_t nsel, double* D2, int* assign, double* d_out,
                        double* dmin = nullptr) {
    // exactly one output: a distance (one centre) or an assignment
    if ((d_out != nullptr) == (assign != nullptr) || (d_out && K != 1) || K < 1 || K > HX_KMAX)
        return cudaErrorInvalidValue;
    k_sk_terms<<<(unsigned)std::min<int64_t>((nsel * K * 4 + 255) / 256, 4096), 256>>>(T, theta, ldt, col0, K, sel,
                                                                                     nsel, D2);
    const size_t smem = (size_t)(2 * SK_STAGE * 4 + 32) * K * sizeof(double);      // at most 101 KB (K = 12)
    cudaError_t e = cudaFuncSetAttribute(k_sk_dist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((2 * SK_STAGE * 4 + 32) * HX_KMAX * sizeof(double)));
    if (e != cudaSuccess) return e;
    k_sk_dist<<<(unsigned)((I + 31) / 32), 32 * K + SK_LOADERS, smem>>>(bed, bps, I, D2, K, sel, nsel, assign, d_out, dmin);
    return cudaGetLastError();
}

// The seed's t-th uniform draw in [0, 1): 53 bits of SplitMix64(seed + t).
double sk_uniform(uint64_t seed, uint64_t t) {
    uint64_t z = seed + t + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

struct SkBuf {   // device buffers of one call, freed on every exit
    std::vector<void*> p;
    ~SkBuf() { for (void* x : p) cudaFree(x); }
    template <class T> cudaError_t get(T** out, size_t n) {
        cudaError_t e = cudaMalloc((void**)out, std::max<size_t>(n, 1) * sizeof(T));
        if (e == cudaSuccess) p.push_back(*out);
        return e;
    }
};

int sk_status(cudaError_t e) {
    return e == cudaSuccess ? HX_OK : (e == cudaErrorMemoryAllocation ? HX_ENOMEM : HX_ECUDA);
}

}  // namespace
}  // namespace hx

#define HX_SK_CK(expr)                          \
    do {                                        \
        cudaError_t e_ = (expr);                \
        if (e_ != cudaSuccess) return hx::sk_status(e_); \
    } while (0)

extern "C" int hx_skfr(const uint8_t* bed, int64_t bytes_per_snp, int64_t n_snp, int64_t I, int32_t K,
                       int64_t sparsity, int32_t max_iter, uint64_t seed, int32_t device, int32_t* clusters,
                       int64_t* aims, int32_t* iters, double* objective) {
    using namespace hx;
    const int64_t M = n_snp - n_snp % 2, nb = M / 2;
    if (!bed || !clusters || !aims || I < 1 || bytes_per_snp < (I + 3) / 4 || n_snp < 2 || max_iter < 1)
        return HX_EINVAL;
    if (K < 1 || K > HX_KMAX) return HX_EUNSUPPORTED;
    if (K > I || sparsity < 1 || sparsity > nb) return HX_EINVAL;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return HX_ECUDA;
    HX_SK_CK(cudaSetDevice(device));
    SkBuf b;
    uint8_t* d_bed = nullptr;
    double *T = nullptr, *theta = nullptr, *score = nullptr, *d2 = nullptr, *n = nullptr;
    int* assign = nullptr;
    int64_t* sel = nullptr;
    uint8_t* keep = nullptr;
    HX_SK_CK(b.get(&d_bed, (size_t)bytes_per_snp * M + 32));   // sk_word reads past the last row's end
    HX_SK_CK(b.get(&T, (size_t)4 * M));
    HX_SK_CK(b.get(&theta, (size_t)M * K));
    HX_SK_CK(b.get(&score, (size_t)M));
    HX_SK_CK(b.get(&d2, (size_t)I));
    HX_SK_CK(b.get(&n, (size_t)K));
    HX_SK_CK(b.get(&assign, (size_t)I));
    HX_SK_CK(b.get(&sel, (size_t)M));
    HX_SK_CK(b.get(&keep, (size_t)M));
    const int64_t W = (I + 15) / 16;
    unsigned* masks = nullptr;
    double* D2 = nullptr;
    HX_SK_CK(b.get(&masks, (size_t)W * K));
    HX_SK_CK(b.get(&D2, (size_t)M * K * 4));
    const unsigned gm = (unsigned)((W * K + 255) / 256);
    HX_SK_CK(cudaMemcpy(d_bed, bed, (size_t)bytes_per_snp * M, cudaMemcpyHostToDevice));
    HX_SK_CK(cudaMemset(theta, 0, (size_t)M * K * sizeof(double)));
    const unsigned gw = (unsigned)((M + SK_WARPS - 1) / SK_WARPS);
    k_sk_masks<<<gm, 256>>>(nullptr, I, W, 1, masks);
    k_sk_tables<<<gw, SK_THREADS>>>(d_bed, bytes_per_snp, W, M, masks, T);
    HX_SK_CK(cudaGetLastError());
    std::vector<int64_t> all(M);
    std::iota(all.begin(), all.end(), (int64_t)0);
    HX_SK_CK(cudaMemcpy(sel, all.data(), (size_t)M * sizeof(int64_t), cudaMemcpyHostToDevice));
    const unsigned gr = (unsigned)std::min<int64_t>((M + 255) / 256, 4096);

    // k-means++ start over all SNPs
    std::vector<double> hd(I), ht(I);
    int64_t c = std::min<int64_t>((int64_t)(sk_uniform(seed, 0) * (double)I), I - 1);
    k_sk_row<<<gr, 256>>>(d_bed, bytes_per_snp, c, T, M, K, 0, theta);
    HX_SK_CK(launch_dist(1, I, d_bed, bytes_per_snp, T, theta, K, 0, sel, M, D2, nullptr, d2));
    HX_SK_CK(cudaMemcpy(hd.data(), d2, (size_t)I * sizeof(double), cudaMemcpyDeviceToHost));
    for (int t = 1; t < K; ++t) {
        std::vector<double> cs(I);
        double acc = 0.0;
        for (int64_t i = 0; i < I; ++i) { acc += hd[i]; cs[i] = acc; }
        const double target = sk_uniform(seed, (uint64_t)t) * acc;
        c = I - 1;
        for (int64_t i = 0; i < I; ++i)
            if (cs[i] > target) { c = i; break; }
        k_sk_row<<<gr, 256>>>(d_bed, bytes_per_snp, c, T, M, K, t, theta);
        HX_SK_CK(launch_dist(1, I, d_bed, bytes_per_snp, T, theta, K, t, sel, M, D2, nullptr, d2));
        HX_SK_CK(cudaMemcpy(ht.data(), d2, (size_t)I * sizeof(double), cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < I; ++i)
            if (ht[i] < hd[i]) hd[i] = ht[i];
    }
    HX_SK_CK(launch_dist(K, I, d_bed, bytes_per_snp, T, theta, K, 0, sel, M, D2, assign, nullptr));
    std::vector<int> ha(I), hn_assign(I);
    HX_SK_CK(cudaMemcpy(ha.data(), assign, (size_t)I * sizeof(int), cudaMemcpyDeviceToHost));

    std::vector<double> hs(M), bs(nb), hn(K);
    std::vector<int64_t> order(nb), kept;
    std::vector<uint8_t> hk(M);
    int it = 0;
    for (it = 1; it <= max_iter; ++it) {
        std::fill(hn.begin(), hn.end(), 0.0);
        for (int64_t i = 0; i < I; ++i) hn[ha[i]] += 1.0;
        HX_SK_CK(cudaMemcpy(n, hn.data(), (size_t)K * sizeof(double), cudaMemcpyHostToDevice));
        k_sk_masks<<<gm, 256>>>(assign, I, W, K, masks);
        k_sk_centers<<<gw, SK_THREADS>>>(d_bed, bytes_per_snp, W, M, K, masks, n, T, theta, score);
        HX_SK_CK(cudaGetLastError());
        HX_SK_CK(cudaMemcpy(hs.data(), score, (size_t)M * sizeof(double), cudaMemcpyDeviceToHost));
        for (int64_t k = 0; k < nb; ++k) bs[k] = hs[2 * k] + hs[2 * k + 1];
        std::iota(order.begin(), order.end(), (int64_t)0);
        // the `sparsity` first in that order, as a set (they are sorted by index next)
        std::nth_element(order.begin(), order.begin() + (sparsity - 1), order.end(),
                         [&](int64_t x, int64_t y) { return bs[x] > bs[y] || (bs[x] == bs[y] && x < y); });
        std::vector<int64_t> kb(order.begin(), order.begin() + sparsity);
        std::sort(kb.begin(), kb.end());
        kept.clear();
        for (int64_t k : kb) { kept.push_back(2 * k); kept.push_back(2 * k + 1); }
        std::fill(hk.begin(), hk.end(), (uint8_t)0);
        for (int64_t l : kept) hk[l] = 1;
        HX_SK_CK(cudaMemcpy(keep, hk.data(), (size_t)M, cudaMemcpyHostToDevice));
        k_sk_mask<<<(unsigned)std::min<int64_t>((M * K + 255) / 256, 4096), 256>>>(theta, keep, M, K);
        HX_SK_CK(cudaGetLastError());
        HX_SK_CK(cudaMemcpy(sel, kept.data(), kept.size() * sizeof(int64_t), cudaMemcpyHostToDevice));
        HX_SK_CK(launch_dist(K, I, d_bed, bytes_per_snp, T, theta, K, 0, sel, (int64_t)kept.size(), D2, assign,
                             nullptr, d2));
        HX_SK_CK(cudaMemcpy(hn_assign.data(), assign, (size_t)I * sizeof(int), cudaMemcpyDeviceToHost));
        const bool changed = hn_assign != ha;
        ha.swap(hn_assign);
        if (!changed) break;
    }
    if (it > max_iter) it = max_iter;
    if (objective) {   // within-cluster sum of squares over the kept SNPs, summed in individual order
        HX_SK_CK(cudaMemcpy(hd.data(), d2, (size_t)I * sizeof(double), cudaMemcpyDeviceToHost));
        double w = 0.0;
        for (int64_t i = 0; i < I; ++i) w += hd[i];
        *objective = w;
    }
    std::copy(ha.begin(), ha.end(), clusters);
    std::copy(kept.begin(), kept.end(), aims);
    if (iters) *iters = it;
    return HX_OK;
}
