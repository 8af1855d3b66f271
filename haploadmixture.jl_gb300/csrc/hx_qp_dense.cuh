// hx_qp_dense.cuh -- batched QP, one warp per problem, dense.
#pragma once
#include "hx_ops.cuh"
#include <climits>

namespace hx {
namespace {
constexpr unsigned QP_FULL = 0xffffffffu;

// Dense active-set QP, one warp per problem: exact minimiser of 0.5 d'Hd - z'd subject to
// lo <= d <= hi and G equality groups (G = 0: none; G = 1: sum d = 0;
// G >= 2: the variables a with a % G == k sum to 0, for every k), by the
// primal active-set method of the oracle (same working-set rules, tie-breaks
// and tolerance).  The free
// block of H is factorised by a warp-parallel right-looking Cholesky in
// shared memory.  Restates OpenADMIXTURE's create_tableau!/quadratic_program!
// contract as called at src/algorithms_inner.jl:160-166, :303-305 and
// :307-310 (the P quartets' K equalities).  The equality form of the P step runs
// on it; the others run on the kernels of hx_qp.cu and come here for problems
// whose free block is not positive definite to rounding (a pivot at its floor).  With G >= 2 the multipliers come
// from the G x G Schur system S nu = E_F y1 + E_X d_X, S = E_F H_FF^-1 E_F',
// and a group's last free variable (fixed by its equality) never blocks.
// GB300's FP64 unit is narrow and every lane's FP64 operation costs issue
// slots on it, so each scalar step (square root, pivot reciprocal, the
// solved unknown of a triangular sweep) is computed by lane 0 alone and
// broadcast; rows then scale by the reciprocal.  The working set may start
// from a previous solve's final set (box-only problems, where any set is a
// feasible start): the method converges to the same unique minimiser.
enum { QF = 0, QL = 1, QH = 2 };

struct QPWork {
    double* A;
    double *d, *z, *lo, *hi, *r, *y1, *y2, *ds, *g, *iv;
    double *Y, *S, *nu, *rhs;   // G >= 2 only: nF x G, G x G, G, G
    int *st, *F;
};

__device__ __forceinline__ double wsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(QP_FULL, v, o);
    return v;
}
__device__ __forceinline__ double wmax(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(QP_FULL, v, o));
    return v;
}

// L L' x = b in place (L lower, iv[a] = 1 / L[a,a]).
__device__ void tri_solve(const double* A, const double* iv, int nF, double* x, int lane) {
    for (int a = 0; a < nF; ++a) {
        __syncwarp();
        double xa = 0.0;
        if (lane == 0) {
            xa = x[a] * iv[a];
            x[a] = xa;
        }
        xa = __shfl_sync(QP_FULL, xa, 0);
        for (int rr = a + 1 + lane; rr < nF; rr += 32) x[rr] -= A[rr + nF * a] * xa;
    }
    for (int a = nF - 1; a >= 0; --a) {
        __syncwarp();
        double xa = 0.0;
        if (lane == 0) {
            xa = x[a] * iv[a];
            x[a] = xa;
        }
        xa = __shfl_sync(QP_FULL, xa, 0);
        for (int rr = lane; rr < a; rr += 32) x[rr] -= A[a + nF * rr] * xa;
    }
    __syncwarp();
}

// L L' X = B in place for the ncol columns of X (nF x ncol, column-major).
__device__ void tri_solve_cols(const double* A, const double* iv, int nF, double* X, int ncol, int lane) {
    for (int a = 0; a < nF; ++a) {
        __syncwarp();
        for (int c = lane; c < ncol; c += 32) X[a + nF * c] *= iv[a];
        __syncwarp();
        const int m = nF - a - 1;
        for (int e = lane; e < m * ncol; e += 32) {
            const int rr = a + 1 + e % m, c = e / m;
            X[rr + nF * c] -= A[rr + nF * a] * X[a + nF * c];
        }
    }
    for (int a = nF - 1; a >= 0; --a) {
        __syncwarp();
        for (int c = lane; c < ncol; c += 32) X[a + nF * c] *= iv[a];
        __syncwarp();
        for (int e = lane; e < a * ncol; e += 32) {
            const int rr = e % a, c = e / a;
            X[rr + nF * c] -= A[a + nF * rr] * X[a + nF * c];
        }
    }
    __syncwarp();
}

// GROUPS: the G-group path (G >= 2, instantiated apart so that the other
// forms keep their register allocation); otherwise G is 0 or 1.
template <bool GROUPS, class HF>
__device__ int warp_qp(int n, int G, const HF& H, const QPWork& w) {
    const int lane = threadIdx.x & 31;
    double zs = 1.0;
    for (int a = lane; a < n; a += 32) zs = fmax(zs, fabs(w.z[a]));
    zs = wmax(zs);
    const double tol = 1e-12 * zs;
    const int max_iter = 4 * n + 20;
    if (GROUPS)
        for (int k = lane; k < G; k += 32) w.nu[k] = 0.0;
    for (int it = 0; it < max_iter; ++it) {
        __syncwarp();
        int nF = 0;
        for (int a = 0; a < n; ++a)
            if (w.st[a] == QF) {
                if (lane == 0) w.F[nF] = a;
                ++nF;
            }
        __syncwarp();
        double nu = 0.0;
        if (nF > 0) {
            for (int a = lane; a < nF; a += 32) {
                const int fa = w.F[a];
                double s = w.z[fa];
                for (int b = 0; b < n; ++b)
                    if (w.st[b] != QF) s -= H(fa, b) * w.d[b];
                w.r[a] = s;
                for (int b = 0; b < nF; ++b) w.A[a + nF * b] = H(fa, w.F[b]);
            }
            __syncwarp();
            double md = 0.0;
            for (int a = lane; a < nF; a += 32) md = fmax(md, fabs(w.A[a + nF * a]));
            md = wmax(md);
            const double fl = 1e-300 + 1e-14 * md;
            for (int c = 0; c < nF; ++c) {
                __syncwarp();
                double inv = 0.0;
                if (lane == 0) {
                    double s = w.A[c + nF * c];
                    if (!(s > fl)) s = fl;
                    const double lcc = sqrt(s);
                    inv = 1.0 / lcc;
                    w.A[c + nF * c] = lcc;
                    w.iv[c] = inv;
                }
                inv = __shfl_sync(QP_FULL, inv, 0);
                for (int rr = c + 1 + lane; rr < nF; rr += 32) w.A[rr + nF * c] *= inv;
                __syncwarp();
                for (int rr = c + 1 + lane; rr < nF; rr += 32) {
                    const double lrc = w.A[rr + nF * c];
                    for (int s2 = c + 1; s2 <= rr; ++s2) w.A[rr + nF * s2] -= lrc * w.A[s2 + nF * c];
                }
            }
            __syncwarp();
            for (int a = lane; a < nF; a += 32) w.y1[a] = w.r[a];
            tri_solve(w.A, w.iv, nF, w.y1, lane);
            if (GROUPS) {
                for (int e = lane; e < nF * G; e += 32) {
                    const int a = e % nF, k = e / nF;
                    w.Y[e] = (w.F[a] % G == k) ? 1.0 : 0.0;
                }
                tri_solve_cols(w.A, w.iv, nF, w.Y, G, lane);
                for (int e = lane; e < G * G; e += 32) {
                    const int k = e % G, l = e / G;
                    double s = 0.0;
                    for (int a = 0; a < nF; ++a)
                        if (w.F[a] % G == k) s += w.Y[a + nF * l];
                    w.S[e] = s;
                }
                for (int k = lane; k < G; k += 32) {
                    double s = 0.0;
                    for (int a = 0; a < nF; ++a)
                        if (w.F[a] % G == k) s += w.y1[a];
                    for (int b = 0; b < n; ++b)
                        if (w.st[b] != QF && b % G == k) s += w.d[b];
                    w.rhs[k] = s;
                }
                __syncwarp();
                if (lane == 0) {   // G x G Cholesky and the two sweeps, as the oracle
                    double* S = w.S;
                    double smax = 0.0;
                    for (int k = 0; k < G; ++k) smax = fmax(smax, fabs(S[k + G * k]));
                    const double sfl = 1e-300 + 1e-14 * smax;
                    for (int c = 0; c < G; ++c) {
                        double s = S[c + G * c];
                        for (int k = 0; k < c; ++k) s -= S[c + G * k] * S[c + G * k];
                        if (!(s > sfl)) s = sfl;
                        const double lcc = sqrt(s);
                        S[c + G * c] = lcc;
                        for (int rr = c + 1; rr < G; ++rr) {
                            double t = S[rr + G * c];
                            for (int k = 0; k < c; ++k) t -= S[rr + G * k] * S[c + G * k];
                            S[rr + G * c] = t / lcc;
                        }
                    }
                    for (int a = 0; a < G; ++a) {
                        double t = w.rhs[a];
                        for (int k = 0; k < a; ++k) t -= S[a + G * k] * w.nu[k];
                        w.nu[a] = t / S[a + G * a];
                    }
                    for (int a = G - 1; a >= 0; --a) {
                        double t = w.nu[a];
                        for (int k = a + 1; k < G; ++k) t -= S[k + G * a] * w.nu[k];
                        w.nu[a] = t / S[a + G * a];
                    }
                }
                __syncwarp();
                for (int a = lane; a < nF; a += 32) {
                    double t = w.y1[a];
                    for (int l = 0; l < G; ++l) t -= w.Y[a + nF * l] * w.nu[l];
                    w.ds[a] = t;
                }
            } else if (G == 1) {
                for (int a = lane; a < nF; a += 32) w.y2[a] = 1.0;
                tri_solve(w.A, w.iv, nF, w.y2, lane);
                double cf = 0.0;
                for (int b = lane; b < n; b += 32)
                    if (w.st[b] != QF) cf -= w.d[b];
                cf = wsum(cf);
                double s1 = 0.0, s2 = 0.0;
                for (int a = lane; a < nF; a += 32) { s1 += w.y1[a]; s2 += w.y2[a]; }
                s1 = wsum(s1);
                s2 = wsum(s2);
                nu = (s1 - cf) / s2;
                for (int a = lane; a < nF; a += 32) w.ds[a] = w.y1[a] - nu * w.y2[a];
            } else {
                for (int a = lane; a < nF; a += 32) w.ds[a] = w.y1[a];
            }
            __syncwarp();
        }
        // ratio test: smallest step ratio < 1, lowest variable index on ties
        double best = 1.0;
        int bidx = INT_MAX, bto = QF;
        for (int a = lane; a < nF; a += 32) {
            const int fa = w.F[a];
            if (GROUPS) {   // a group's last free variable is fixed by its equality
                int cnt = 0;
                for (int b = 0; b < nF; ++b) cnt += (w.F[b] % G == fa % G);
                if (cnt == 1) continue;
            }
            const double s = w.ds[a] - w.d[fa];
            double ra = 2.0;
            int to = QF;
            if (s < 0.0) { ra = (w.lo[fa] - w.d[fa]) / s; to = QL; }
            else if (s > 0.0) { ra = (w.hi[fa] - w.d[fa]) / s; to = QH; }
            if (ra < best) { best = ra; bidx = fa; bto = to; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(QP_FULL, best, o);
            const int oi = __shfl_xor_sync(QP_FULL, bidx, o);
            const int ot = __shfl_xor_sync(QP_FULL, bto, o);
            if (ob < best || (ob == best && oi < bidx)) { best = ob; bidx = oi; bto = ot; }
        }
        if (bidx == INT_MAX) {
            for (int a = lane; a < nF; a += 32) w.d[w.F[a]] = w.ds[a];
            __syncwarp();
            for (int a = lane; a < n; a += 32) {
                double s = -w.z[a];
                for (int b = 0; b < n; ++b) s += H(a, b) * w.d[b];
                w.g[a] = s + (GROUPS ? w.nu[a % G] : nu);
            }
            __syncwarp();
            double wv = tol;
            int rel = INT_MAX;
            for (int a = lane; a < n; a += 32) {
                if (w.lo[a] >= 0.0 && w.hi[a] <= 0.0) continue;
                double v = 0.0;
                if (w.st[a] == QL) v = -w.g[a];
                else if (w.st[a] == QH) v = w.g[a];
                if (v > wv) { wv = v; rel = a; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(QP_FULL, wv, o);
                const int oi = __shfl_xor_sync(QP_FULL, rel, o);
                if (ov > wv || (ov == wv && oi < rel)) { wv = ov; rel = oi; }
            }
            if (rel == INT_MAX) return it + 1;
            __syncwarp();
            if (lane == 0) w.st[rel] = QF;
        } else {
            const double al = best < 0.0 ? 0.0 : best;
            for (int a = lane; a < nF; a += 32) {
                const int fa = w.F[a];
                w.d[fa] = w.d[fa] + al * (w.ds[a] - w.d[fa]);
            }
            __syncwarp();
            if (lane == 0) {
                w.d[bidx] = (bto == QL) ? w.lo[bidx] : w.hi[bidx];
                w.st[bidx] = bto;
            }
        }
    }
    return -1;
}

// Per-warp workspace for problems of up to nmax variables and gmax >= 2
// equality groups (gmax = 0 when the problems have at most one equality).
__device__ QPWork carve(double* base, int nmax, int gmax = 0) {
    QPWork w;
    w.A = base;
    double* v = base + nmax * nmax;
    w.d = v; w.z = v + nmax; w.lo = v + 2 * nmax; w.hi = v + 3 * nmax; w.r = v + 4 * nmax;
    w.y1 = v + 5 * nmax; w.y2 = v + 6 * nmax; w.ds = v + 7 * nmax; w.g = v + 8 * nmax; w.iv = v + 9 * nmax;
    double* e = v + 10 * nmax;
    w.Y = e; w.S = e + nmax * gmax; w.nu = w.S + gmax * gmax; w.rhs = w.nu + gmax;
    w.st = reinterpret_cast<int*>(w.rhs + gmax);
    w.F = w.st + nmax;
    return w;
}
__host__ __device__ constexpr size_t qp_warp_bytes(int nmax, int gmax = 0) {
    return (size_t)(nmax * nmax + 10 * nmax + nmax * gmax + gmax * gmax + 2 * gmax) * sizeof(double) +
           (size_t)(2 * nmax) * sizeof(int);
}

struct HQ {
    const double* X;
    int K;
    double pen;   // penalty form: rho on every entry (rho * 1 1'); 0 in the equality form
    __device__ double operator()(int r, int c) const { return X[r + K * c] + pen; }
};
struct HP {
    const double* X;   // XtX_p + K*K*4j
    int K;
    double rho;
    __device__ double operator()(int r, int c) const {
        const int l = r / K, k2 = r - l * K, l2 = c / K, k = c - l2 * K;
        return (l == l2 ? X[(int64_t)K * K * l + k2 + K * k] : 0.0) + (k2 == k ? rho : 0.0);
    }
};

}  // namespace
}  // namespace hx
