// hx_qp.cu -- batched simplex-constrained QPs of the Q step and of the P step's
// penalty form (src/algorithms_inner.jl:134-168, 264-305).
//
// Exact minimiser of 0.5 d'Hd - z'd, lo <= d <= hi (and sum d = 0 on the Q
// side), by the primal active-set method of the oracle: solve on the free
// variables (Cholesky factor of the free block), step to the first bound met
// (lowest index on ties), and when no bound is met release the bound with the
// largest multiplier.  An FP64 operation of a warp takes 64 clocks of its quarter of
// an SM, however few of its lanes work and whether or not the next one waits for
// it, so both kernels keep the lanes full: the Q side solves one problem per lane,
// the P side one per group of K lanes; and the pivots' roots and all comparisons
// (FP64 operations too) are done in integers.  P side, 20,000 blocks at K = 10:
// 2.10 ms with 16 lanes per problem, 1.50 with 10, 1.27 with the integer forms;
// 4,000 blocks at K = 5: 0.59, 0.45, 0.39.  Both perform, element by element, the operations of
// the dense factorisation and sweeps of the free block in index order, and leave
// out only those whose operands are exact zeros, so the results do not depend
// on this arrangement (the mixed method rounds them to FP32 afterwards, which
// would turn a last-bit difference into one of 6e-8).  A free block that is not
// positive definite to rounding (fewer data than variables, or a mixed-precision
// Hessian whose entries span more than its 16 bits) has pivots at their floor; what
// follows grows, and where it overflows, the zeros of fixed variables meet infinities
// that the dense solver never forms: such a problem is handed to it by its warp and
// solved from the start.  (Every floored pivot went there once, one after another:
// 20,000 problems of rank 1, K = 8, Q side: 6.9 ms, 1.9 here.)
// Calls of few problems and P steps of a handful of individuals go to the dense solver
// as a whole, a warp per problem (see the launchers).
#include "hx_ops.cuh"
#include "hx_qp_dense.cuh"
#include "hx_tc.cuh"
#include <climits>

namespace hx {
namespace {
using tc::tri_idx;
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ bool finite(double x) { return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000; }
// x > f for f > 0
__device__ __forceinline__ bool above(double x, double f) {
    const long long b = __double_as_longlong(x);
    return b > __double_as_longlong(f) && b <= 0x7FF0000000000000ll;
}
__device__ __forceinline__ long long abs_bits(double x) { return __double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFll; }
constexpr long long INF_BITS = 0x7FF0000000000000ll;
// The larger of two magnitudes, as bits
__device__ __forceinline__ long long max_bits(long long a, long long b) { return a > b ? a : b; }
// x > 0, and x < 0
__device__ __forceinline__ bool positive(double x) { return __double_as_longlong(x) > 0 && abs_bits(x) <= INF_BITS; }
__device__ __forceinline__ bool negative(double x) {
    return __double2hiint(x) < 0 && abs_bits(x) > 0 && abs_bits(x) <= INF_BITS;
}
// |a| < |b|
__device__ __forceinline__ bool smaller(double a, double b) { return abs_bits(a) < abs_bits(b) && abs_bits(b) <= INF_BITS; }
// Whether the step s from d passes the bound ahead (upper bound 1 - v, lower 0 - v):
// a ratio num / s below 1, or a bound passed by rounding, before dividing
__device__ __forceinline__ bool passes(double s, double v, double d, bool& upw, double& num) {
    upw = positive(s);
    num = ((upw ? 1.0 : 0.0) - v) - d;
    return abs_bits(s) != 0 && (smaller(num, s) || (upw ? negative(num) : positive(num)));
}

// ------------------------------------------------------------------ Q side
// One problem per thread, its K x K triangle in shared memory (entry e of
// thread t at e * QQ_LD + t), factor and vectors in registers.  Rows and
// columns of fixed variables are zero in the factor, so the code has no
// data-dependent indices.
constexpr int QQ_THREADS = 64, QQ_LD = QQ_THREADS + 1;

// One problem on the dense solver, by a whole warp; base: K^2 + 11 K doubles of
// shared memory.
__device__ __noinline__ void qp_q_dense(int K, int64_t pr, const double* XtX, const double* Xtz, const double* q,
                                        double* qdiff, double* slots, double pen_rho, double* base) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    QPWork w = carve(base, K);
    for (int a = lane; a < K; a += 32) {
        const double qa = q[(int64_t)K * pr + a];
        w.d[a] = 0.0;
        w.z[a] = Xtz[(int64_t)K * pr + a];
        w.lo[a] = 0.0 - qa;
        w.hi[a] = 1.0 - qa;
        w.st[a] = (w.lo[a] >= 0.0 && w.hi[a] <= 0.0) ? QL : QF;
    }
    __syncwarp();
    HQ H{XtX + (int64_t)K * K * pr, K, pen_rho >= 0.0 ? pen_rho : 0.0};
    const int it = warp_qp<false>(K, pen_rho < 0.0 ? 1 : 0, H, w);
    __syncwarp();
    for (int a = lane; a < K; a += 32) qdiff[(int64_t)K * pr + a] = w.d[a];
    if (it < 0 && lane == 0) atomicAdd(slots + S_QP_FAIL, 1.0);
    __syncwarp();
}

// Sum of the elements of x (K <= 12) in the order of a butterfly over 16 lanes.
template <int K> __device__ __forceinline__ double tree_sum(const double (&x)[K]) {
    double t8[8], t4[4];
#pragma unroll
    for (int a = 0; a < 8; ++a) t8[a] = (a < K ? x[a < K ? a : 0] : 0.0) + (a + 8 < K ? x[a + 8 < K ? a + 8 : 0] : 0.0);
#pragma unroll
    for (int a = 0; a < 4; ++a) t4[a] = t8[a] + t8[a + 4];
    return (t4[0] + t4[2]) + (t4[1] + t4[3]);
}

template <int K>
__global__ void __launch_bounds__(QQ_THREADS)
k_qp_q(int64_t n, const double* __restrict__ XtX, const double* __restrict__ Xtz, const double* __restrict__ q,
       double* __restrict__ qdiff, double* slots, double pen_rho) {
    constexpr int NT = K * (K + 1) / 2;
    __shared__ double sH[NT * QQ_LD];
    __shared__ double sX[K * QQ_THREADS];        // per warp: ranks, then the dense solver's work
    const int tid = threadIdx.x;
    const int64_t p0 = (int64_t)blockIdx.x * QQ_THREADS, pr = p0 + tid;
    const int np = (int)min((int64_t)QQ_THREADS, n - p0);
    const bool eq = pen_rho < 0.0;               // equality form, else rho on every entry
    for (int t = tid; t < np * K * K; t += QQ_THREADS) {
        const int x = t / (K * K), e = t - x * K * K, c = e / K, r = e - c * K;
        if (r >= c) sH[tri_idx<K>(c, r) * QQ_LD + x] = XtX[p0 * K * K + t] + (eq ? 0.0 : pen_rho);
    }
    __syncthreads();
    const bool mine = tid < np;
    const double* H = sH + (mine ? tid : 0);
    double* xs = sX + (tid >> 5) * 32 * K + (tid & 31);
    auto h = [&](int a, int b) { return H[(a <= b ? tri_idx<K>(a, b) : tri_idx<K>(b, a)) * QQ_LD]; };
    // Sum over the free variables as the list of them is summed: element of rank
    // r in place r of the butterfly.
    auto free_sum = [&](const double (&x)[K], unsigned fr) {
        double y[K];
        if (fr == (1u << K) - 1u) return tree_sum<K>(x);
#pragma unroll
        for (int a = 0; a < K; ++a) xs[a * 32] = 0.0;
#pragma unroll
        for (int a = 0; a < K; ++a)
            if ((fr >> a) & 1u) xs[__popc(fr & ((1u << a) - 1u)) * 32] = x[a];
#pragma unroll
        for (int a = 0; a < K; ++a) y[a] = xs[a * 32];
        return tree_sum<K>(y);
    };
    double z[K], d[K], qa[K];
    unsigned fr = 0u, up = 0u, no = 0u;          // free; at the upper bound; both bounds at 0
    double tol = 1.0;
#pragma unroll
    for (int a = 0; a < K; ++a) {
        qa[a] = mine ? q[pr * K + a] : 0.0;
        z[a] = mine ? Xtz[pr * K + a] : 0.0;
        tol = fmax(tol, fabs(z[a]));
        d[a] = 0.0;
        if (0.0 - qa[a] >= 0.0 && 1.0 - qa[a] <= 0.0) no |= 1u << a;
        else fr |= 1u << a;
    }
    tol *= 1e-12;
    const int max_iter = 4 * K + 20;
    bool done = !mine, over = false;
#pragma unroll 1
    for (int it = 0; it < max_iter && !done; ++it) {
        double A[NT], y[K], o[K];
        long long mb = 0;
#pragma unroll
        for (int a = 0; a < K; ++a) {
            const bool fa = (fr >> a) & 1u;
            double s = z[a];
            if (fr != (1u << K) - 1u) {
#pragma unroll
                for (int b = 0; b < K; ++b)
                    if (!((fr >> b) & 1u)) s = fma(-h(a, b), d[b], s);
            }
            y[a] = fa ? s : 0.0;
            o[a] = fa ? 1.0 : 0.0;
#pragma unroll
            for (int b = a; b < K; ++b) A[tri_idx<K>(a, b)] = fa && ((fr >> b) & 1u) ? h(a, b) : 0.0;
            mb = max_bits(mb, abs_bits(A[tri_idx<K>(a, a)]));
        }
        const double fl = 1e-300 + 1e-14 * __longlong_as_double(mb);
        // A = L L': entry (a, b), b > a, ends as L[b, a]; y and o follow through
        // the forward sweep
        double iv[K];
#pragma unroll
        for (int a = 0; a < K; ++a) {
            const double pv = A[tri_idx<K>(a, a)];
            const bool fa = (fr >> a) & 1u;
            iv[a] = fa ? inv_root(above(pv, fl) ? pv : fl) : 0.0;
            y[a] *= iv[a];
            o[a] *= iv[a];
#pragma unroll
            for (int b = a + 1; b < K; ++b) A[tri_idx<K>(a, b)] *= iv[a];
#pragma unroll
            for (int b = a + 1; b < K; ++b) {
                const double l = A[tri_idx<K>(a, b)];
#pragma unroll
                for (int c = b; c < K; ++c)
                    A[tri_idx<K>(b, c)] = fma(-l, A[tri_idx<K>(a, c)], A[tri_idx<K>(b, c)]);
                y[b] = fma(-l, y[a], y[b]);
                o[b] = fma(-l, o[a], o[b]);
            }
        }
#pragma unroll
        for (int a = K - 1; a >= 0; --a) {
            y[a] *= iv[a];
            o[a] *= iv[a];
#pragma unroll
            for (int b = 0; b < a; ++b) {
                y[b] = fma(-A[tri_idx<K>(b, a)], y[a], y[b]);
                o[b] = fma(-A[tri_idx<K>(b, a)], o[a], o[b]);
            }
        }
        double nu = 0.0;
        if (eq && fr) {
            double f[K];
#pragma unroll
            for (int a = 0; a < K; ++a) f[a] = (fr >> a) & 1u ? 0.0 : -d[a];
            nu = (free_sum(y, fr) - tree_sum<K>(f)) / free_sum(o, fr);
        }
        // y becomes the target of the free variables
        double best = 1.0;
        int bi = -1;
        bool bup = false;
#pragma unroll
        for (int a = 0; a < K; ++a) {
            if (!((fr >> a) & 1u)) { y[a] = d[a]; continue; }
            if (eq) y[a] = fma(-nu, o[a], y[a]);
            over |= !finite(y[a]);
            const double s = y[a] - d[a];
            bool u;
            double num;
            if (passes(s, qa[a], d[a], u, num)) {
                const double ra = num / s;
                if (ra < best) { best = ra; bi = a; bup = u; }
            }
        }
        if (over) break;
        if (bi < 0) {
#pragma unroll
            for (int a = 0; a < K; ++a) d[a] = y[a];
            double wv = tol;
            int rel = -1;
            if ((fr | no) != (1u << K) - 1u) {
#pragma unroll
                for (int a = 0; a < K; ++a) {
                    if (((fr | no) >> a) & 1u) continue;
                    double g = -z[a];
#pragma unroll
                    for (int b = 0; b < K; ++b) g = fma(h(a, b), d[b], g);
                    g += nu;
                    const double v = (up >> a) & 1u ? g : -g;
                    if (above(v, wv)) { wv = v; rel = a; }
                }
            }
            if (rel < 0) { done = true; break; }
            fr |= 1u << rel;
        } else {
            const double al = best < 0.0 ? 0.0 : best;
#pragma unroll
            for (int a = 0; a < K; ++a) {
                if ((fr >> a) & 1u) d[a] = fma(al, y[a] - d[a], d[a]);
                if (a == bi) d[a] = bup ? 1.0 - qa[a] : 0.0 - qa[a];
            }
            fr &= ~(1u << bi);
            up = bup ? up | (1u << bi) : up & ~(1u << bi);
        }
    }
    if (mine && !over) {
#pragma unroll
        for (int a = 0; a < K; ++a) qdiff[pr * K + a] = d[a];
        if (!done) atomicAdd(slots + S_QP_FAIL, 1.0);
    }
    unsigned left = __ballot_sync(FULL, over);
    while (left) {
        const int b = __ffs(left) - 1;
        left &= left - 1;
        qp_q_dense(K, pr - (tid & 31) + b, XtX, Xtz, q, qdiff, slots, pen_rho, sX + (tid >> 5) * 32 * K);
    }
}

// ------------------------------------------------------------------ P side
// Variables (h, k), H = blockdiag(D_0 .. D_3) + rho on equal k.  In the dense
// factorisation of the free block (order h, then k), the rows of all later
// haplotypes are alike left of them: before column (h, .) every block
// (h', h''), h'' >= h, h' > h'', is one and the same K x K matrix T (rho I at
// first), and so are the rows V of L that haplotype h's columns leave in it.  So
// the factor takes, per haplotype, its own K x K block, V once, and the update
// by V V' of T and of the later diagonal blocks: about K^3 x 5 operations
// instead of 11 K^3.
// One problem per group of K lanes; lane k holds row k of each block and the
// four variables (h, k).
template <int K> struct PDim {
    static constexpr int PW = 32 / K;                       // problems per warp
    static constexpr int WARPS = 2;
    // per problem (doubles): D [4][K][K], L [4][K][K], V [3][K][K], iv [4][K], vec [4][K]
    static constexpr int RAW = 11 * K * K + 8 * K;
    // problems of a warp start in different banks
    static constexpr int LD = (RAW + 15) / 16 * 16 + (K % 4 == 0 ? 4 : K);
    static constexpr size_t SMEM = (size_t)WARPS * PW * LD * sizeof(double);
    static_assert(PW * LD >= 16 * K * K + 44 * K, "a warp's memory holds the dense solver's work");
};

// One block on the dense solver, by a whole warp; base: 16 K^2 + 44 K doubles.
__device__ __noinline__ void qp_p_dense(int K, int64_t j, const double* XtX, const double* Xtz, const double* p,
                                        double rho, double* pdiff, double* slots, int8_t* ws, double* base) {
    const int lane = threadIdx.x & 31, nv = 4 * K;
    __syncwarp();
    QPWork w = carve(base, nv);
    for (int a = lane; a < nv; a += 32) {
        const double pa = p[(int64_t)nv * j + a];
        w.d[a] = 0.0;
        w.z[a] = Xtz[(int64_t)nv * j + a];
        w.lo[a] = 0.0 - pa;
        w.hi[a] = 1.0 - pa;
        int s0 = ws ? (int)ws[(int64_t)nv * j + a] : QF;
        if (w.lo[a] >= 0.0 && w.hi[a] <= 0.0) s0 = QL;
        w.st[a] = s0;
        w.d[a] = s0 == QL ? w.lo[a] : (s0 == QH ? w.hi[a] : 0.0);
    }
    __syncwarp();
    HP H{XtX + (int64_t)K * K * 4 * j, K, rho};
    const int it = warp_qp<false>(nv, 0, H, w);
    __syncwarp();
    for (int a = lane; a < nv; a += 32) {
        pdiff[(int64_t)nv * j + a] = w.d[a];
        if (ws) ws[(int64_t)nv * j + a] = (int8_t)w.st[a];
    }
    if (it < 0 && lane == 0) atomicAdd(slots + S_QP_FAIL, 1.0);
    __syncwarp();
}

template <int K>
__global__ void __launch_bounds__(32 * PDim<K>::WARPS)
k_qp_p4(int64_t n, const double* __restrict__ XtX, const double* __restrict__ Xtz, const double* __restrict__ p,
        double rho, double* __restrict__ pdiff, double* slots, int8_t* __restrict__ ws) {
    using P = PDim<K>;
    constexpr int KK = K * K;
    extern __shared__ double smem_p[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = min(lane / K, P::PW - 1), k = lane - g * K, base = g * K;     // k >= K: idle lane
    const int64_t j = ((int64_t)blockIdx.x * P::WARPS + warp) * P::PW + g;
    const bool valid = j < n;
    const bool row = k < K;
    const int kc = row ? k : K - 1;                 // index for loads of idle lanes
    double* D = smem_p + (warp * P::PW + g) * P::LD;   // H(k, b) of block h at h KK + b K + k
    double* L = D + 4 * KK;                         // L[s, c] of block h at h KK + c K + s
    double* V = L + 4 * KK;                         // V[k, c] of block h at h KK + c K + k
    double* iv = V + 3 * KK;                        // reciprocal roots of the pivots (0: fixed)
    double* vec = iv + 4 * K;
    if (row) for (int t = k; t < 4 * KK; t += K) D[t] = valid ? XtX[j * 4 * KK + t] : (t % KK / K == t % K ? 1.0 : 0.0);
    // lane o places on in the group, round its end: ceil(log2 K) such steps reach every lane
    auto next = [&](int o) { return base + (row ? k + o - (k + o < K ? 0 : K) : o); };
    double z[4], d[4], pa[4];
    unsigned fr = 0u, up = 0u, no = 0u;             // bits h: free; at the upper bound; both bounds at 0
    double zs = 1.0;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const int64_t at = (j * 4 + h) * K + kc;
        pa[h] = valid ? p[at] : 0.25;
        z[h] = valid ? Xtz[at] : 0.0;
        d[h] = 0.0;
        if (row) {
            zs = fmax(zs, fabs(z[h]));
            // warm start from the previous solve's working set (bounds only: feasible)
            int s0 = ws && valid ? (int)ws[at] : 0;
            if (0.0 - pa[h] >= 0.0 && 1.0 - pa[h] <= 0.0) { no |= 1u << h; s0 = 1; }
            if (s0 == 0) fr |= 1u << h;
            if (s0 == 2) up |= 1u << h;
            d[h] = s0 == 1 ? 0.0 - pa[h] : (s0 == 2 ? 1.0 - pa[h] : 0.0);
        }
    }
#pragma unroll
    for (int o = 1; o < K; o *= 2) zs = fmax(zs, __shfl_sync(FULL, zs, next(o)));
    const double tol = 1e-12 * zs;
    const int max_iter = 16 * K + 20;
    __syncwarp();
    double dk[4];                                   // diagonal of H
#pragma unroll
    for (int h = 0; h < 4; ++h) dk[h] = D[h * KK + kc * K + kc] + rho;
    bool done = !valid, over = false;               // over: left to the dense solver
#pragma unroll 1
    for (int it = 0; it < max_iter; ++it) {
        if (__all_sync(FULL, done)) break;
        __syncwarp();
        // fixed variables to vec (free ones 0), largest free diagonal
        long long mb = 0;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const bool f = (fr >> h) & 1u;
            if (row) vec[h * K + k] = f ? 0.0 : d[h];
            if (row && f) mb = max_bits(mb, abs_bits(dk[h]));
        }
#pragma unroll
        for (int o = 1; o < K; o *= 2) mb = max_bits(mb, __shfl_sync(FULL, mb, next(o)));
        const double fl = 1e-300 + 1e-14 * __longlong_as_double(mb);
        __syncwarp();
        // right-hand sides z - H d over the fixed variables, in index order
        double x[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            double s = z[h];
            if (!__all_sync(FULL, !row || done || fr == 0xFu)) {
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l != h) {
                        s = fma(-rho, (fr >> l) & 1u ? 0.0 : d[l], s);
                    } else {
#pragma unroll
                        for (int b = 0; b < K; ++b) s = fma(-D[h * KK + b * K + kc], vec[h * K + b], s);
                    }
                }
            }
            x[h] = row && ((fr >> h) & 1u) ? s : 0.0;
        }
        // factorisation, forward sweep alongside.  One copy of the code serves the
        // four haplotypes, with C, the later blocks G and the right-hand sides
        // moved up by one after each (written out four times, the loop was 210 KB
        // of code at K = 10, and 6% slower)
        double T[K], C[K], G[3][K];                  // row k of T, of this and of the later diagonal blocks
#pragma unroll
        for (int a = 0; a < K; ++a) {
            T[a] = a == k ? rho : 0.0;
            const int at = a <= kc ? a * K + kc : kc * K + a;
            C[a] = a == k ? dk[0] : D[at];
#pragma unroll
            for (int h = 1; h < 4; ++h) G[h - 1][a] = a == k ? dk[h] : D[h * KK + at];
        }
        __syncwarp();
#pragma unroll 1
        for (int h = 0; h < 4; ++h) {
            double *Lh = L + h * KK, *Vh = V + h * KK;
            const bool f = row && ((fr >> h) & 1u);
            const unsigned fm = __ballot_sync(FULL, f) >> base;          // free indices of this problem's h
            double M[K], W[K];
#pragma unroll
            for (int a = 0; a < K; ++a) {
                M[a] = f && ((fm >> a) & 1u) ? C[a] : 0.0;
                W[a] = T[a];
            }
#pragma unroll
            for (int c = 0; c < K; ++c) {
                const double pv = __shfl_sync(FULL, M[c], base + c);
                const double ivc = (fm >> c) & 1u ? inv_root(above(pv, fl) ? pv : fl) : 0.0;
                const double l = k > c ? M[c] * ivc : 0.0;
                if (row) Lh[c * K + k] = l;
                if (k == c) iv[h * K + c] = ivc;
                const double xa = __shfl_sync(FULL, x[0], base + c) * ivc;
                x[0] = k == c ? xa : fma(-l, xa, x[0]);
                W[c] *= ivc;                          // V[k, c]
                __syncwarp();
#pragma unroll
                for (int s = c + 1; s < K; ++s) {
                    const double ls = Lh[c * K + s];
                    M[s] = fma(-l, ls, M[s]);
                    W[s] = fma(-W[c], ls, W[s]);
                }
            }
            if (row) vec[h * K + k] = x[0];
            if (h == 3) break;
            if (row) {
#pragma unroll
                for (int c = 0; c < K; ++c) Vh[c * K + k] = W[c];
            }
            __syncwarp();
#pragma unroll 1
            for (int c = 0; c < K; ++c) {
                const double w = -Vh[c * K + kc], xa = vec[h * K + c];
                const double* v = Vh + c * K;
                x[1] = fma(w, xa, x[1]);
#pragma unroll
                for (int a = 0; a < K; ++a) G[0][a] = fma(w, v[a], G[0][a]);
                if (h < 2) {
                    x[2] = fma(w, xa, x[2]);
#pragma unroll
                    for (int a = 0; a < K; ++a) {
                        T[a] = fma(w, v[a], T[a]);
                        G[1][a] = fma(w, v[a], G[1][a]);
                    }
                }
                if (h == 0) {
                    x[3] = fma(w, xa, x[3]);
#pragma unroll
                    for (int a = 0; a < K; ++a) G[2][a] = fma(w, v[a], G[2][a]);
                }
            }
#pragma unroll
            for (int a = 0; a < K; ++a) {
                C[a] = G[0][a];
                G[0][a] = G[1][a];
                G[1][a] = G[2][a];
            }
            // rows of fixed variables get sums too; the masks leave them unused
            x[0] = (fr >> (h + 1)) & 1u ? x[1] : 0.0;
            x[1] = (fr >> (h + 2)) & 1u ? x[2] : 0.0;
            x[2] = (fr >> (h + 3)) & 1u ? x[3] : 0.0;
        }
        __syncwarp();
        // backward sweep, the same way: x[b] belongs to haplotype h - b
#pragma unroll
        for (int b = 0; b < 4; ++b) x[b] = vec[(3 - b) * K + kc];
#pragma unroll 1
        for (int h = 3; h >= 0; --h) {
            const double *Lh = L + h * KK, *Vh = V + h * KK;
#pragma unroll
            for (int c = K - 1; c >= 0; --c) {
                const double xa = __shfl_sync(FULL, x[0], base + c) * iv[h * K + c];
                x[0] = k == c ? xa : (k < c ? fma(-Lh[kc * K + c], xa, x[0]) : x[0]);
            }
            __syncwarp();
            if (row) vec[h * K + k] = x[0];
            __syncwarp();
#pragma unroll 1
            for (int c = K - 1; c >= 0; --c) {
                const double xa = vec[h * K + c];
                const double* v = Vh + kc * K + c;
                if (h > 0) x[1] = fma(-v[-KK], xa, x[1]);
                if (h > 1) x[2] = fma(-v[-2 * KK], xa, x[2]);
                if (h > 2) x[3] = fma(-v[-3 * KK], xa, x[3]);
            }
#pragma unroll
            for (int b = 0; b < 3; ++b) x[b] = x[b + 1];
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) x[h] = vec[h * K + kc];
        bool inf = false;
#pragma unroll
        for (int h = 0; h < 4; ++h) inf |= row && ((fr >> h) & 1u) && !finite(x[h]);
        if (((__ballot_sync(FULL, inf) >> base) & ((1u << K) - 1u)) && !done) { over = true; done = true; }
        // targets; ratio test: smallest step ratio < 1, lowest variable index (h, k) on ties
        double best = 1.0;
        int bidx = INT_MAX;
        bool bup = false;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            if (!(row && ((fr >> h) & 1u))) { x[h] = d[h]; continue; }
            const double s = x[h] - d[h];
            bool upw;
            double num;
            if (passes(s, pa[h], d[h], upw, num)) {
                const double ra = num / s;
                if (ra < best) { best = ra; bidx = h * K + k; bup = upw; }
            }
        }
        long long bb = __double_as_longlong(best);       // as an integer in the same order
        if (bb < 0) bb = abs_bits(best) == 0 ? 0 : bb ^ 0x7FFFFFFFFFFFFFFFll;
        int bto = bup ? 1 : 0;
#pragma unroll
        for (int o = 1; o < K; o *= 2) {
            const long long ob = __shfl_sync(FULL, bb, next(o));
            const int oi = __shfl_sync(FULL, bidx, next(o)), ot = __shfl_sync(FULL, bto, next(o));
            if (ob < bb || (ob == bb && oi < bidx)) { bb = ob; bidx = oi; bto = ot; }
        }
        const bool blocked = bidx != INT_MAX;
        if (!done && blocked) {
            const double al = bb < 0 ? 0.0 : __longlong_as_double(bb);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if ((fr >> h) & 1u) d[h] = fma(al, x[h] - d[h], d[h]);
                if (row && bidx == h * K + k) {
                    d[h] = bto ? 1.0 - pa[h] : 0.0 - pa[h];
                    fr &= ~(1u << h);
                    up = bto ? up | (1u << h) : up & ~(1u << h);
                }
            }
        }
        // no bound met: take the point, release the largest multiplier
        if (!done && !blocked) {
#pragma unroll
            for (int h = 0; h < 4; ++h) d[h] = x[h];
        }
        if (__all_sync(FULL, done || blocked)) continue;
        __syncwarp();
        if (row) {
#pragma unroll
            for (int h = 0; h < 4; ++h) vec[h * K + k] = d[h];
        }
        __syncwarp();
        double wv = tol;
        int rel = INT_MAX;
        if (row && !done && !blocked) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                if (((fr | no) >> h) & 1u) continue;
                double gr = -z[h];
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l != h) {
                        gr = fma(rho, d[l], gr);
                    } else {
#pragma unroll
                        for (int b = 0; b < K; ++b)
                            gr = fma(b == k ? dk[h] : D[h * KK + b * K + kc], vec[h * K + b], gr);
                    }
                }
                const double v = (up >> h) & 1u ? gr : -gr;
                if (above(v, wv)) { wv = v; rel = h * K + k; }
            }
        }
#pragma unroll
        for (int o = 1; o < K; o *= 2) {
            const double ov = __shfl_sync(FULL, wv, next(o));
            const int oi = __shfl_sync(FULL, rel, next(o));
            const long long bo = __double_as_longlong(ov), bw = __double_as_longlong(wv);    // tol or above
            if (bo > bw || (bo == bw && oi < rel)) { wv = ov; rel = oi; }
        }
        if (!done && !blocked) {
            if (rel == INT_MAX) done = true;
            else if (rel % K == k && row) fr |= 1u << (rel / K);
        }
    }
    if (valid && row && !over) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int64_t at = (j * 4 + h) * K + k;
            pdiff[at] = d[h];
            if (ws) ws[at] = (fr >> h) & 1u ? 0 : ((up >> h) & 1u ? 2 : 1);
        }
    }
    if (valid && !done && k == 0) atomicAdd(slots + S_QP_FAIL, 1.0);
    unsigned left = __ballot_sync(FULL, over && k == 0);
    while (left) {
        const int b = __ffs(left) - 1;
        left &= left - 1;
        qp_p_dense(K, __shfl_sync(FULL, j, b), XtX, Xtz, p, rho, pdiff, slots, ws, smem_p + warp * P::PW * P::LD);
    }
}

// ------------------------------------------------------------------ dense
// All problems of a call on the dense solver, a warp each.
constexpr int QD_WARPS = 4;
template <bool PS>
__global__ void __launch_bounds__(32 * QD_WARPS)
k_qp_dense(int K, int64_t n, const double* __restrict__ XtX, const double* __restrict__ Xtz, const double* __restrict__ x,
           double rho, double* __restrict__ diff, double* slots, int8_t* __restrict__ ws) {
    extern __shared__ double smem_d[];
    const int warp = threadIdx.x >> 5;
    const int64_t t = (int64_t)blockIdx.x * QD_WARPS + warp;
    if (t >= n) return;
    double* base = smem_d + warp * (qp_warp_bytes(PS ? 4 * K : K) / sizeof(double));
    if (PS) qp_p_dense(K, t, XtX, Xtz, x, rho, diff, slots, ws, base);
    else qp_q_dense(K, t, XtX, Xtz, x, diff, slots, rho, base);
}
template <bool PS>
cudaError_t launch_dense(int K, int64_t n, const double* XtX, const double* Xtz, const double* x, double rho, double* diff,
                         double* slots, int8_t* ws, cudaStream_t st) {
    k_qp_dense<PS><<<(unsigned)((n + QD_WARPS - 1) / QD_WARPS), 32 * QD_WARPS, QD_WARPS * qp_warp_bytes(PS ? 4 * K : K),
                     st>>>(K, n, XtX, Xtz, x, rho, diff, slots, ws);
    return cudaGetLastError();
}

#define HX_FOR_K(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)
}  // namespace

// A lane's solve takes as long for one problem as for 20,000, and goes through all K
// variables however many are fixed; the dense solver's time grows with the problems and
// shrinks with the variables that are fixed.  It is ahead, for the whole Q step, where
// blocks are fewer than variables (many bounds met one after another; 2 blocks, K = 5:
// 0.45 -> 0.34 ms at 2,000 individuals, 0.48 -> 0.67 at 10,000; K = 8: 1.05 -> 0.72 at
// 4,000, 1.13 -> 1.53 at 10,000; K = 3 the same at 2,000), and from K = 11 on for small
// cohorts (500 blocks, K = 12: 0.46 -> 0.37 ms at 500 individuals, 0.82 -> 0.78 at 3,000,
// the same at 4,000; 2,750 problems, K = 11: 0.70 -> 0.67; K = 8: 0.21 ms both at 1,000).
// The results are the same bits.
cudaError_t launch_qp_q(int K, int64_t n, int64_t J, const double* XtX, const double* Xtz, const double* q, double* qdiff,
                        double* slots, cudaStream_t st, double pen_rho) {
    if (J < K ? K >= 4 && n <= 500 * K : K >= 11 && n <= 250 * K)
        return launch_dense<false>(K, n, XtX, Xtz, q, pen_rho, qdiff, slots, nullptr, st);
    const unsigned g = (unsigned)((n + QQ_THREADS - 1) / QQ_THREADS);
#define HX_CASE(KK) case KK: k_qp_q<KK><<<g, QQ_THREADS, 0, st>>>(n, XtX, Xtz, q, qdiff, slots, pen_rho); break;
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
    return cudaGetLastError();
}

cudaError_t init_qp_attrs(int K) {
    cudaError_t e = cudaFuncSetAttribute(k_qp_dense<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(QD_WARPS * qp_warp_bytes(4 * HX_KMAX)));
    if (e != cudaSuccess) return e;
#define HX_CASE(KK)                                                                                     \
    case KK:                                                                                            \
        return cudaFuncSetAttribute(k_qp_p4<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PDim<KK>::SMEM);
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
}

// With fewer than 2 K individuals most variables end at bounds, met one after another
// (see launch_qp_q): whole P step of 5 individuals x 1,000 blocks, dense against K lanes,
// K = 5: 3.9 and 6.8 ms, K = 8: 11.3 and 25.7, K = 12: 37.6 and 58.8; of 24 individuals x
// 10,000 blocks, K = 8: 11.9 and 6.0.
cudaError_t launch_qp_p_pen(int K, int64_t n, int64_t I, const double* XtX, const double* Xtz, const double* p, double rho,
                            double* pdiff, double* slots, int8_t* ws, cudaStream_t st) {
    if (K >= 4 && I < 2 * K) return launch_dense<true>(K, n, XtX, Xtz, p, rho, pdiff, slots, ws, st);
#define HX_CASE(KK)                                                                                              \
    case KK: {                                                                                                   \
        constexpr int per = PDim<KK>::WARPS * PDim<KK>::PW;                                                      \
        k_qp_p4<KK><<<(unsigned)((n + per - 1) / per), 32 * PDim<KK>::WARPS, PDim<KK>::SMEM, st>>>(              \
            n, XtX, Xtz, p, rho, pdiff, slots, ws);                                                              \
        break;                                                                                                   \
    }
    switch (K) { HX_FOR_K(HX_CASE) default: return cudaErrorInvalidValue; }
#undef HX_CASE
    return cudaGetLastError();
}

}  // namespace hx
