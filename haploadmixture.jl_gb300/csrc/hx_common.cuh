// hx_common.cuh -- shared definitions of the GB300 HaploADMIXTURE fitting path.
//
// Genotype layout in HBM ("class words"): after hx_create the PLINK BED bytes
// are decoded once into one 32-bit word per (individual, group of 8 two-SNP
// blocks): word G[jw * Ipad + i] holds in nibble b (bits 4b..4b+3) the class
// of block j = 8*jw + b for individual i, as code(SNP 2j) | code(SNP 2j+1) << 2
// with the raw 2-bit BED codes (0b00 hom A1, 0b01 missing, 0b10 het, 0b11 hom
// A2; src/loops.jl:55-71).  Padding individuals (i >= I) and padding blocks
// (j >= J) carry nibble 0x5 (both SNPs missing), whose likelihood factor is 1
// and whose expected counts are 0, so padding never contributes.  The layout
// keeps the BED's 4 bits per (i, j) pair and turns every pass into fully
// coalesced word loads along individuals.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#define HX_KMAX 12
#define HX_QMAX_DEV 6
#define HX_IPAD 128
#define HX_PAD_NIBBLE 0x5u
#define HX_PAD_WORD 0x55555555u

namespace hx {

// Genotype value of a raw BED code (src/loops.jl:64-71): 0->0, 1->missing(3), 2->1, 3->2.
__host__ __device__ constexpr int code_g(int c) { return c == 0 ? 0 : (c == 1 ? 3 : (c == 2 ? 1 : 2)); }

// Haplotype-set masks of a class (bit h for haplotype h = 2*allele(SNP1)+allele(SNP2)).
// The pair likelihood is L = F1 * F2 with F_s = sum_{h in S_s} qp_h, except the
// double heterozygote (L = qp00 qp11 + qp01 qp10, both phases) and the
// double-missing class (L = 1).  This is the factored form of
// @coefs_likelihood (src/loops.jl:85-104): F1 = a1 + a2 and F2 = b1 + b2.
__host__ __device__ constexpr unsigned class_m1(unsigned nib) {
    int g1 = code_g(nib & 3), g2 = code_g((nib >> 2) & 3);
    if (g1 == 3 && g2 == 3) return 0;
    if (g1 == 1 && g2 == 1) return 0;
    if (g1 == 3) return g2 == 2 ? 0xAu : 0x5u;          // {01,11} : {00,10}
    if (g2 == 3) return g1 == 2 ? 0xCu : 0x3u;          // {10,11} : {00,01}
    int s1 = g1 == 2 ? 1 : 0, s2 = g2 == 2 ? 1 : 0;     // first copy
    return 1u << (2 * s1 + s2);
}
__host__ __device__ constexpr unsigned class_m2(unsigned nib) {
    int g1 = code_g(nib & 3), g2 = code_g((nib >> 2) & 3);
    if (g1 == 3 && g2 == 3) return 0;
    if (g1 == 1 && g2 == 1) return 0;
    if (g1 == 3) return g2 == 0 ? 0x5u : 0xAu;          // second copy's SNP2 allele
    if (g2 == 3) return g1 == 0 ? 0x3u : 0xCu;
    int s1 = g1 >= 1 ? 1 : 0, s2 = g2 >= 1 ? 1 : 0;     // second copy
    return 1u << (2 * s1 + s2);
}
__host__ __device__ constexpr uint64_t make_tab(bool second) {
    uint64_t t = 0;
    for (unsigned n = 0; n < 16; ++n) t |= (uint64_t)(second ? class_m2(n) : class_m1(n)) << (4 * n);
    return t;
}
constexpr uint64_t TAB_M1 = make_tab(false);
constexpr uint64_t TAB_M2 = make_tab(true);
constexpr unsigned NIB_HH = 2u | (2u << 2);   // het / het
constexpr unsigned NIB_MM = 1u | (1u << 2);   // missing / missing

template <typename T> __device__ __forceinline__ T rcp(T x);
template <> __device__ __forceinline__ float rcp<float>(float x) { return __frcp_rn(x); }
template <> __device__ __forceinline__ double rcp<double>(double x) { return 1.0 / x; }

// 1/x in fixed point, to 0.5001 ulp: from the hardware's FP32 reciprocal y of the
// significand m cut to 24 bits, one step y (1 + e + e^2), e = 1 - m y < 2^-22 (the
// cubically convergent form of Newton's iteration; e, from the low 64 bits of the
// product, is exact), and one rounding.  About 30 integer operations, which find free
// issue slots where an FP64 operation takes 64 clocks of its quarter of an SM: the
// same step in FP64 was 3 of the K + 4 operations per item of the plain passes,
// and those were what bound them.  Outside 2^-1000 .. 2^1000 (zeros, NaN,
// infinities) and below zero it divides, out of line.
static __device__ __noinline__ double rcp64_edge(double x) { return 1.0 / x; }
__device__ __forceinline__ double rcp64(double x) {
    typedef long long i64;
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), ex = hi >> 20;
    if (ex - 23u > 2000u) return rcp64_edge(x);
    float y0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0)
        : "f"(__uint_as_float(0x3F800000u | ((hi & 0xFFFFFu) << 3) | (lo >> 29))));
    const unsigned Y = (__float_as_uint(fminf(y0, 0x1.fffffep-1f)) << 7) ^ 0xC0000000u;    // y 2^31
    const unsigned long long m = ((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;   // 2^52
    const i64 e = -(i64)(m * Y);                                // 2^83
    const int e1 = (int)(e >> 37);                              // 2^46
    const i64 d = e + (((i64)e1 * e1) >> 9);                    // e + e^2, 2^83
    const i64 c = (i64)(int)(d >> 32) * Y + __umulhi((unsigned)d, Y);    // y d, 2^82
    const i64 r = (i64)((unsigned long long)Y << 22) + ((c + (1ll << 28)) >> 29);          // 2^53 / m
    return __longlong_as_double(r + ((i64)(2044u - ex) << 52));
}

// 1 / sqrt(s) as the QPs' factorisation uses it: the reciprocal of the rounded root,
// both correctly rounded.  In fixed point: with s = m 4^k, 1 <= m < 4, one
// cubically convergent step y (1 + e/2 + 3 e^2/8), e = 1 - m y^2, from the
// hardware's FP32 reciprocal root leaves y ~ 1 / sqrt(m) within 2^-53, and
// G ~ sqrt(m) = m y; the remainders m - G^2 and 1 - G R, exact in the low 64 bits
// of the products, then tell how far G and R are from the nearest 53-bit numbers
// (1 and 2 units at most).  Outside 2^-600 .. 2^600 the operators, out of line.
static __device__ __noinline__ double inv_root_edge(double s) { return 1.0 / sqrt(s); }
__device__ __forceinline__ double inv_root(double s) {
    typedef unsigned long long u64;
    typedef long long i64;
    const int hi = __double2hiint(s);
    if (((unsigned)hi >> 20) - 423u > 1200u) return inv_root_edge(s);
    const int ex = (hi >> 20) - 1023, odd = ex & 1, half = (ex - odd) >> 1;
    const u64 b = ((u64)__double_as_longlong(s) & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const u64 m = b << (10 + odd);                                     // m 2^62
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__uint2float_rn((unsigned)(m >> 32)) * 0x1p-30f));
    const unsigned Y0 = __float2uint_rz(y0 * 0x1p31f);                 // y 2^31, at most 2^31 (1 + 2^-22)
    const i64 e = (i64)((1ull << 60) - __umul64hi(m, (u64)Y0 * Y0));   // 2^60, |e| < 2^39
    const int e1 = (int)(e >> 24);                                     // 2^36
    const i64 t = (e >> 1) + (((i64)e1 * e1 * 3) >> 15);               // e/2 + 3 e^2/8, 2^60
    const int t1 = (int)((t + 64) >> 7);                               // 2^53
    const u64 y = ((u64)Y0 << 31) + (u64)(((i64)Y0 * t1) >> 22);       // 2^62
    u64 G = (__umul64hi(m, y) + 128) >> 8;                             // sqrt(m) 2^52
    const i64 r = (i64)((m << 42) - G * G);
    G = G + (r > (i64)G) - (r <= -(i64)G);
    u64 R = (y + 256) >> 9;                                            // 2^53 / sqrt(m)
    const i64 g = (i64)G, q = -2 * (i64)(R * G);                       // 2 (2^105 - R G)
    R = R + (q > g) + (q > 3 * g) - (q < -g) - (q < -3 * g);
    return __longlong_as_double((i64)(R + ((u64)(1021 - half) << 52)));
}

// Per-pair evaluation.  Given the class nibble and the mixed haplotype
// frequencies qp[h] = sum_k q[k,i] p[k,4j+h] it returns
//   L    : the pair likelihood (src/loops.jl:85-104, 254),
//   u[h] : c_h / qp_h = d log L / d qp_h, with c_h the E-step expected
//          haplotype counts of @coefs (src/loops.jl:114-155).
// Branch-free: the class only selects operands.
template <typename T>
__device__ __forceinline__ void pair_eval(unsigned nib, const T qp[4], T& L, T u[4]) {
    const unsigned m1 = (unsigned)(TAB_M1 >> (4 * nib)) & 0xFu;
    const unsigned m2 = (unsigned)(TAB_M2 >> (4 * nib)) & 0xFu;
    T F1 = ((((m1 & 1u) ? qp[0] : T(0)) + ((m1 & 2u) ? qp[1] : T(0))) + ((m1 & 4u) ? qp[2] : T(0))) +
           ((m1 & 8u) ? qp[3] : T(0));
    T F2 = ((((m2 & 1u) ? qp[0] : T(0)) + ((m2 & 2u) ? qp[1] : T(0))) + ((m2 & 4u) ? qp[2] : T(0))) +
           ((m2 & 8u) ? qp[3] : T(0));
    const bool hh = nib == NIB_HH;
    const bool mm = nib == NIB_MM;
    T den = qp[0] * qp[3] + qp[1] * qp[2];
    F1 = hh ? den : F1;
    F1 = mm ? T(1) : F1;
    F2 = (hh || mm) ? T(1) : F2;
    const T r1 = rcp<T>(F1), r2 = rcp<T>(F2);
    L = F1 * F2;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        T a = ((m1 >> h) & 1u) ? r1 : T(0);
        T b = ((m2 >> h) & 1u) ? r2 : T(0);
        T v = a + b;
        u[h] = hh ? qp[3 - h] * r1 : v;
    }
}

// Copy-level allele indicators of a raw SNP code, as FP32 0/1 values
// {copy 1 may carry allele 0, copy 1 allele 1, copy 2 allele 0, copy 2 allele 1}:
// hom A1 (code 0) {0}{0}; missing (1) {0,1}{0,1}; het (2) {0}{1}; hom A2 (3) {1}{1}.
// With M[a][b] = qp_{2a+b}, F_s = sum_{a in A_s, b in B_s} M[a][b] over the
// copy-s sets of the block's two SNPs, which is the class_m1/class_m2 factor
// for every class except the double heterozygote and double missing.
// A kernel keeps the table in shared memory (snp_table_init by its first 16
// threads, then a barrier) and reads one 16-byte row per SNP: the four rows
// occupy distinct banks, so a warp's lookups never conflict.
__device__ __forceinline__ void snp_table_init(float4* tab, int tid) {
    if (tid < 16) {
        const int c = tid >> 2, e = tid & 3;
        const int bits = c == 0 ? 0x5 : c == 1 ? 0xF : c == 2 ? 0x9 : 0xA;   // bit e: indicator e
        reinterpret_cast<float*>(tab)[tid] = (bits >> e) & 1 ? 1.f : 0.f;
    }
}

// FP32 pair evaluation for the mixed method: same results as pair_eval<float>
// (L identical; u to the last bit of an approximate reciprocal), with the class
// turned into arithmetic on indicator rows instead of per-haplotype selects.
__device__ __forceinline__ void pair_eval_tab(unsigned nib, const float qp[4], float& L, float u[4], const float4* tab) {
    const float4 ta = tab[nib & 3u], tb = tab[(nib >> 2) & 3u];
    const float v10 = fmaf(tb.y, qp[1], tb.x * qp[0]), v11 = fmaf(tb.y, qp[3], tb.x * qp[2]);
    const float v20 = fmaf(tb.w, qp[1], tb.z * qp[0]), v21 = fmaf(tb.w, qp[3], tb.z * qp[2]);
    float F1 = fmaf(ta.y, v11, ta.x * v10);
    float F2 = fmaf(ta.w, v21, ta.z * v20);
    const bool hh = nib == NIB_HH;
    const bool mm = nib == NIB_MM;
    const float den = fmaf(qp[1], qp[2], qp[0] * qp[3]);
    F1 = hh ? den : F1;
    F1 = mm ? 1.f : F1;
    F2 = (hh || mm) ? 1.f : F2;
    L = F1 * F2;
    float r1, r2;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(F1));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2) : "f"(F2));
    const float hr = hh ? r1 : 0.f;
    r1 = (hh || mm) ? 0.f : r1;
    r2 = (hh || mm) ? 0.f : r2;
    const float x10 = ta.x * r1, x11 = ta.y * r1, x20 = ta.z * r2, x21 = ta.w * r2;
    u[0] = fmaf(hr, qp[3], fmaf(x10, tb.x, x20 * tb.z));
    u[1] = fmaf(hr, qp[2], fmaf(x10, tb.y, x20 * tb.w));
    u[2] = fmaf(hr, qp[1], fmaf(x11, tb.x, x21 * tb.z));
    u[3] = fmaf(hr, qp[0], fmaf(x11, tb.y, x21 * tb.w));
}

// Likelihood only.
__device__ __forceinline__ float pair_lik_tab(unsigned nib, const float qp[4], const float4* tab) {
    const float4 ta = tab[nib & 3u], tb = tab[(nib >> 2) & 3u];
    const float v10 = fmaf(tb.y, qp[1], tb.x * qp[0]), v11 = fmaf(tb.y, qp[3], tb.x * qp[2]);
    const float v20 = fmaf(tb.w, qp[1], tb.z * qp[0]), v21 = fmaf(tb.w, qp[3], tb.z * qp[2]);
    float F1 = fmaf(ta.y, v11, ta.x * v10);
    float F2 = fmaf(ta.w, v21, ta.z * v20);
    const bool hh = nib == NIB_HH;
    const bool mm = nib == NIB_MM;
    const float den = fmaf(qp[1], qp[2], qp[0] * qp[3]);
    F1 = hh ? den : F1;
    F1 = mm ? 1.f : F1;
    F2 = (hh || mm) ? 1.f : F2;
    return F1 * F2;
}

// Type-generic entry: FP32 uses the indicator table, FP64 the exact select form.
__device__ __forceinline__ void pair_eval_t(unsigned nib, const float qp[4], float& L, float u[4], const float4* tab) {
    pair_eval_tab(nib, qp, L, u, tab);
}
__device__ __forceinline__ void pair_eval_t(unsigned nib, const double qp[4], double& L, double u[4], const float4*) {
    pair_eval<double>(nib, qp, L, u);
}

// Packed FP32x2 arithmetic (sm_100+): fma.rn.f32x2 performs two IEEE FMAs,
// lane by lane, with the results of two fmaf calls.
__device__ __forceinline__ uint64_t f2_dup(float x) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ void f2_split(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// Class rows: for each class the membership of the four haplotypes in the first
// copy's set (class_m1, bytes 0-3) and in the second copy's (class_m2, bytes
// 4-7), 0x40 or 0: the byte as the top byte of a float is 2.0f or 0.0f.  Sixteen
// rows of 8 bytes fill the 32 banks once, so a warp's lookups never conflict and
// take two wavefronts (FP32 rows of 16 bytes took about eleven, and shared-memory
// wavefronts were what bound the P pass and the log-likelihood: 80% of the
// clocks).  Kept in shared memory (cls_table_init by the first 32 threads, then a
// barrier); a row is addressed by 8 * class.
__device__ __forceinline__ void cls_table_init(uint32_t* tab, int tid) {
    if (tid < 32) {
        const unsigned nib = tid >> 1;
        const unsigned m = (unsigned)((tid & 1 ? TAB_M2 : TAB_M1) >> (4 * nib)) & 0xFu;
        tab[tid] = (m & 1u ? 0x40u : 0u) | (m & 2u ? 0x4000u : 0u) | (m & 4u ? 0x400000u : 0u) | (m & 8u ? 0x40000000u : 0u);
    }
}
struct ClsRow { uint64_t a01, a23, b01, b23; };   // 2.0f or 0.0f: first copy's set, second copy's
__device__ __forceinline__ ClsRow cls_row(const uint32_t* tab, unsigned off) {
    const uint2 r = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(tab) + off);
    auto f = [](uint32_t x, unsigned sel) { return __uint_as_float(__byte_perm(x, 0u, sel)); };
    ClsRow c;
    c.a01 = f2_pack(f(r.x, 0x0444), f(r.x, 0x1444));
    c.a23 = f2_pack(f(r.x, 0x2444), f(r.x, 0x3444));
    c.b01 = f2_pack(f(r.y, 0x0444), f(r.y, 0x1444));
    c.b23 = f2_pack(f(r.y, 0x2444), f(r.y, 0x3444));
    return c;
}
// Twice the two copies' factors F1, F2 (0 for the double heterozygote and double
// missing).
__device__ __forceinline__ void cls_factors(const ClsRow& c, uint64_t z01, uint64_t z23, float& F1, float& F2) {
    float a, b;
    f2_split(f2_fma(c.a23, z23, f2_mul(c.a01, z01)), a, b);
    F1 = a + b;
    f2_split(f2_fma(c.b23, z23, f2_mul(c.b01, z01)), a, b);
    F2 = a + b;
}

// scale * u (scale a power of two) of the class at byte offset off = 8 * class,
// from packed (qp0, qp1), (qp2, qp3), in packed FP32x2 arithmetic: the same
// results as pair_eval_tab's u * scale, bit for bit (a copy's set has at most
// two members, so each factor rounds once in either order of the sum; the
// powers of two are exact: 2 / (2 F)).  The double heterozygote takes its operands
// (qp3, qp2, qp1, qp0) / den in the place of the first copy's row.
__device__ __forceinline__ void pair_u_cls(unsigned off, uint64_t z01, uint64_t z23, uint64_t& u01, uint64_t& u23,
                                           const uint32_t* tab, float scale) {
    const ClsRow c = cls_row(tab, off);
    float q0, q1, q2, q3, F1, F2;
    f2_split(z01, q0, q1);
    f2_split(z23, q2, q3);
    cls_factors(c, z01, z23, F1, F2);
    const bool hh = off == 8u * NIB_HH, mm = off == 8u * NIB_MM;
    const float den = fmaf(q1, q2, q0 * q3);
    F1 = hh ? den : F1;
    F1 = mm ? 1.f : F1;
    F2 = hh || mm ? 1.f : F2;
    float r1, r2;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(F1));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2) : "f"(F2));
    const uint64_t r1d = f2_dup(r1 * scale), r2d = f2_dup(r2 * scale);
    float x0, x1, x2, x3;
    f2_split(c.a01, x0, x1);
    f2_split(c.a23, x2, x3);
    const uint64_t s01 = f2_pack(hh ? q3 : x0, hh ? q2 : x1), s23 = f2_pack(hh ? q1 : x2, hh ? q0 : x3);
    u01 = f2_fma(s01, r1d, f2_mul(c.b01, r2d));
    u23 = f2_fma(s23, r1d, f2_mul(c.b23, r2d));
}

// Exact exponent/mantissa split used to accumulate products of likelihoods
// without underflow (one log per CTA instead of two per pair).
__device__ __forceinline__ float renorm(float m, int& e) {
    unsigned b = __float_as_uint(m);
    e += (int)((b >> 23) & 0xFFu) - 127;
    return __uint_as_float((b & 0x007FFFFFu) | 0x3F800000u);
}
__device__ __forceinline__ double renorm(double m, int& e) {
    unsigned long long b = (unsigned long long)__double_as_longlong(m);
    e += (int)((b >> 52) & 0x7FFull) - 1023;
    return __longlong_as_double((long long)((b & 0x000FFFFFFFFFFFFFull) | 0x3FF0000000000000ull));
}

}  // namespace hx
