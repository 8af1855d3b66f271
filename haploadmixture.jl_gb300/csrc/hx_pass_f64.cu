// hx_pass_f64.cu -- the plain method's log-likelihood (src/loops.jl:236-258),
// from the class words or straight from BED bytes.
#include "hx_ops.cuh"
#include "hx_items.cuh"

#define HX_FOR_K(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

namespace hx {
namespace {

constexpr int L_THREADS = 128;
constexpr int L_WARPS = L_THREADS / 32;

template <int K> struct LDim {
    static constexpr int KS = K | 1;                         // row stride (doubles): odd, so rows differ in banks
    static constexpr size_t SMEM = (size_t)(128 + 32) * KS * 8 + (size_t)L_WARPS * 512 * (8 + 2);
};

// CTA: 128 individuals x a chunk of word columns (8 blocks each); warp w:
// individuals 32 w .. +31, four blocks of the column at a time (at most 37 KB of
// shared memory: no attribute to set before a launch).  The
// pair likelihood is a product of mixed frequencies qp for every class but the
// double heterozygote and those with one SNP missing, so a needed item's qp
// multiplies straight into the running product of whichever lane evaluates it
// (homozygous pairs, whose qp counts twice, into one of their own); the other
// classes are finished from the listed qp's.  Products are exponent-
// renormalised: one log per CTA.  Bound by the FP64 unit: K + 1
// operations per needed haplotype (2 of 4 on average) against 4 K + 20 per
// pair before.  BED: the two codes of each block are read from the BED bytes.
template <int K, bool BED>
__global__ void __launch_bounds__(L_THREADS)
k_loglik64(PassArgs a, const uint8_t* __restrict__ bed, int64_t bps) {
    constexpr int KS = LDim<K>::KS;
    extern __shared__ __align__(16) double sm[];
    double* fix = sm;                         // [128][KS] q rows
    double* sp = fix + 128 * KS;              // [32][KS] p rows of the word column
    double* qpb = sp + 32 * KS;               // [WARPS][16][32] qp of the pairs to finish
    uint16_t* lists = reinterpret_cast<uint16_t*>(qpb + L_WARPS * 512);
    __shared__ double red[L_WARPS];
    __shared__ long long rex[L_WARPS];
    __shared__ int rfl[L_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5;
    const unsigned lane = tid & 31, lt = (1u << lane) - 1u;
    const int64_t i0 = (int64_t)blockIdx.x * 128, i = i0 + 32 * warp + lane;
    const int w0 = blockIdx.y * a.per_chunk, w1 = min(a.JW, w0 + a.per_chunk);
    for (int t = tid; t < 128 * K; t += L_THREADS) {
        const int r = t / K, k = t - r * K;
        fix[r * KS + k] = i0 + r < a.I ? a.q[(i0 + r) * K + k] : 0.25;
    }
    const double* qrow = fix + 32 * warp * KS;
    double* qb = qpb + warp * 512;
    uint16_t* list = lists + warp * 512;
    double m1 = 1.0, m2 = 1.0;                // products of qp's that count once / twice
    int e1 = 0, e2 = 0;
    bool zero = false, bad = false;
    auto times = [&](double v, bool twice) {
        // v > 0 in integers: a comparison takes an FP64 operation's time
        const long long vb = __double_as_longlong(v);
        if ((unsigned long long)(vb - 1) >= 0x7FF0000000000000ull) {
            if ((vb << 1) == 0) zero = true; else bad = true;
            v = 1.0;
        }
        int e = 0;
        const double m = renorm((twice ? m2 : m1) * v, e);
        if (twice) { m2 = m; e2 += e; } else { m1 = m; e1 += e; }
    };
    constexpr int PER = (32 * K + L_THREADS - 1) / L_THREADS;
    double nxt[PER];
    auto fetch = [&](int w) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int64_t g = (int64_t)w * 32 * K + u * L_THREADS + tid;
            nxt[u] = u * L_THREADS + tid < 32 * K && g < a.J * 4 * K ? a.p[g] : 0.25;
        }
    };
    uint32_t word = 0;                        // the lane's class word
    auto classes = [&](int w) {
        word = HX_PAD_WORD;
        if (BED) {
            if (i < a.I) {
                word = 0;
                const int64_t j = 8 * (int64_t)w;
#pragma unroll
                for (int b = 0; b < 16; ++b)
                    word |= (j + (b >> 1) < a.J ? (bed[(2 * j + b) * bps + (i >> 2)] >> (2 * (i & 3))) & 3u : 1u) << (2 * b);
            }
        } else {
            word = a.G[(int64_t)w * a.Ipad + i];
        }
    };
    if (w0 < w1) { fetch(w0); classes(w0); }
    for (int w = w0; w < w1; ++w) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int t = u * L_THREADS + tid;
            if (t < 32 * K) sp[t / K * KS + t % K] = nxt[u];
        }
        __syncthreads();
        uint32_t cls = word;
        if (w + 1 < w1) { fetch(w + 1); classes(w + 1); }
#pragma unroll 1
        for (int hb = 0; hb < 2; ++hb, cls >>= 16) {
            const double* prow = sp + 16 * hb * KS;
            int n = 0;
            unsigned cpl = 0;
#pragma unroll
            for (int bb = 0; bb < 4; ++bb) {
                const unsigned nib = (cls >> (4 * bb)) & 0xFu;
                const unsigned need = (unsigned)(TAB_NEED >> (4 * nib)) & 0xFu;
                const unsigned cx = (TAB_CPLX >> nib) & 1u;
                cpl |= cx << bb;
                const unsigned tag = lane | (__popc(need) == 1 ? 512u : 0u) | (cx ? 1024u : 0u);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const bool has = (need >> h) & 1u;
                    const unsigned bal = __ballot_sync(0xffffffffu, has);
                    if (has) list[n + __popc(bal & lt)] = (uint16_t)(tag | ((4 * bb + h) << 5));
                    n += __popc(bal);
                }
            }
            __syncwarp();
#pragma unroll 1
            for (int base = 0; base < n; base += 32) {
                if (base + (int)lane < n) {
                    const unsigned it = list[base + lane];
                    const double* q = qrow + (it & 31u) * KS;
                    const double* p = prow + ((it >> 5) & 15u) * KS;
                    double s = q[0] * p[0];
#pragma unroll
                    for (int k = 1; k < K; ++k) s = fma(q[k], p[k], s);
                    if (it & 1024u) qb[it & 511u] = s;
                    else times(s, it & 512u);
                }
            }
            __syncwarp();
            int nc = 0;
#pragma unroll
            for (int bb = 0; bb < 4; ++bb) {
                const bool has = (cpl >> bb) & 1u;
                const unsigned bal = __ballot_sync(0xffffffffu, has);
                if (has) list[nc + __popc(bal & lt)] = (uint16_t)(lane | (bb << 5) | (((cls >> (4 * bb)) & 0xFu) << 7));
                nc += __popc(bal);
            }
            __syncwarp();
#pragma unroll 1
            for (int base = 0; base < nc; base += 32) {
                if (base + (int)lane < nc) {
                    const unsigned it = list[base + lane], nib = it >> 7;
                    const double* x = qb + ((it >> 5) & 3u) * 128 + (it & 31u);
                    const unsigned need = (unsigned)(TAB_NEED >> (4 * nib)) & 0xFu;
                    if (nib == NIB_HH) {
                        times(fma(x[0], x[96], x[32] * x[64]), false);
                    } else {
                        // one SNP missing: each copy's factor sums the two haplotypes it may be
                        const bool s1 = (nib & 3u) == 1u;
                        const int ib = s1 ? 64 : 32, ic = s1 ? 32 : 64;
                        const bool ab = need & 1u, cd = (need >> (ic >> 5)) & 1u;
                        const double f1 = ab ? x[0] + x[ib] : x[ic] + x[96];
                        const double f2 = ab && cd ? x[ic] + x[96] : f1;
                        times(f1 * f2, false);
                    }
                }
            }
            __syncwarp();
        }
    }
    // the CTA's product, exponents apart, and one log (a log is some 40 FP64
    // operations, more than a short chunk's own work when every lane takes two)
    long long ex = (long long)e1 + 2ll * e2;
    double m = m2;
    auto mul = [&](double y) {
        int e = 0;
        m = renorm(m * y, e);
        ex += e;
    };
    mul(m2);
    mul(m1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, m, o);
        ex += __shfl_xor_sync(0xffffffffu, ex, o);
        mul(y);
    }
    const bool any_zero = __any_sync(0xffffffffu, zero), any_bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        red[warp] = m;
        rex[warp] = ex;
        rfl[warp] = (any_zero ? 1 : 0) | (any_bad ? 2 : 0);
    }
    __syncthreads();
    if (tid == 0) {
        int fl = rfl[0];
        for (int x = 1; x < L_WARPS; ++x) {
            mul(red[x]);
            ex += rex[x];
            fl |= rfl[x];
        }
        double v = log(m) + (double)ex * 0.69314718055994530942;
        if (fl & 1) v = -INFINITY;
        if (fl & 2) v = NAN;
        a.part[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = v;
    }
}

template <int K, bool BED>
cudaError_t run(const PassArgs& a, const uint8_t* bed, int64_t bps, cudaStream_t st) {
    static_assert(LDim<K>::SMEM <= 48 * 1024, "dynamic shared memory without an attribute");
    dim3 grid((unsigned)((a.I + 127) / 128), (unsigned)a.S);
    k_loglik64<K, BED><<<grid, L_THREADS, LDim<K>::SMEM, st>>>(a, bed, bps);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_loglik_f64(int K, const PassArgs& a, cudaStream_t st) {
#define HX_CASE(KK) case KK: return run<KK, false>(a, nullptr, 0, st);
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
}
cudaError_t launch_loglik_f64_bed(int K, const PassArgs& a, const uint8_t* bed, int64_t bps, cudaStream_t st) {
#define HX_CASE(KK) case KK: return run<KK, true>(a, bed, bps, st);
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
}

}  // namespace hx
