// hx_f64.cuh -- the plain (FP64) method's gradient and Hessian passes.
//
// GB300's FP64 units do 2 operations per clock and SM, 1/64 of the FP32
// rate (a warp's operation takes 64 clocks of its quarter of an SM, however few lanes
// work), so a pass that does its K(K+1)/2 accumulations per haplotype there
// costs 90 to 160 clocks per (individual, block) pair (K = 5 .. 8).  These
// passes keep on the FP64 unit only what has to be there, and only for the
// haplotypes that a pair's genotypes allow (1.8 of 4 on average):
//   qp_h = sum_k q[k,i] p[k,4j+h] and the pair's weights, from r_h = 1 / qp_h
//   (which rcp64 forms in integers),
//   W_h = c_h r_h^2 (Hessian) or U_h = c_h r_h (gradient only),
// and form the sums H = sum W v v' (v = p on the Q side, q on the P side;
// src/loops.jl:328-403) exactly on the tensor cores: the error-free splitting
// of Ozaki, Ogita, Oishi and Rump (2012).  Each index's vector is scaled by a power of
// two 2^-f, 2^f its largest entry (Q side) or its sum (P side, 1), rounded up, and W by
// 2^2f (2^f in the gradient-only form), which leaves W' = c_h (2^f / qp_h)^2: c_h at
// least, and not much more even for rare haplotypes; on the P side the row's power of
// two 2^g (its largest frequency) is a third factor, for the same reason.  W' is rounded
// to a multiple of 2^-56 and written as ND_A = 9 signed base-256 digits, the scaled
// products v_k v_k2 to a multiple of 2^-86 as ND_B = 11 digits.  Digits are integers in
// [-128, 127], exact in FP16; a digit product is at most 2^14, and an FP32 accumulator
// column takes at most 9 digit pairs x 96 reduction indices x 2^14 < 2^24 before it is
// read out, so every accumulation is exact.  Digit pairs (a, b) of equal order a + b
// share a column; orders 0 .. 12 are kept (an order-13 pair weighs 2^-88 at most, with
// either sign).  The columns are read out to 128-bit integers, so a chunk's sum does not
// depend on any order; only the chunk sums and the last digits' cut are rounded.
//
// Which inputs: entries of Q and P in [2^-17, 1] (2^-34 without the Hessian), as a fit
// has them; the general passes of hx_pass.cuh take all others (F_LO_HESS).  A product is
// then at least 2^-34 and keeps 53 bits of its own, so that an entry made of small
// products only (all carriers floored in both ancestries) is as accurate as an FP64 sum;
// with 8 digits and 10 orders such entries had 24 to 27 bits.  A double heterozygote's c
// can be small (2^-17): its W' keeps 40 bits then, and with units of 2^-52 the sums of
// cohorts of 30 and 60 individuals were off by up to 4e-13.
//
// The gradient needs no sums of its own beside the Hessian: sum_k2 H[k,k2] x_k2
// = sum W v_k qp = sum U v_k = g_k (x = the row's own vector, qp = v . x), all
// terms of one sign, formed by the reduction of the chunks.
//
// A scaled weight of 2^14 or more (an observed haplotype about 100 times rarer in the
// individual's mixture than in one of the ancestries; 2^38 at most) does not fit the
// digits: its products are added in fixed point to 64-bit integers in global memory
// (order-independent, as every integer sum).
#pragma once
#include "hx_ops.cuh"
#include "hx_tc.cuh"
#include "hx_items.cuh"

namespace hx {
namespace {
using namespace tc;

constexpr int F_GEN_WARPS = 16;                       // generator warps
constexpr int F_THREADS = 32 * (F_GEN_WARPS + 1);     // + one warp that loads and issues
constexpr int F_KD = 32;                              // reduction indices per stage
constexpr int F_RING = 3;                             // vectors and class words of the next stages
constexpr int F_BRING = 2;                            // B tiles: read by the MMAs only, a stage later
constexpr int F_WIN = 3;                              // stages per read-out (96 reduction indices)
constexpr int F_SA = 56, F_SB = 86;                   // units 2^-SA of W', 2^-SB of the products
constexpr long long F_BUDGET = 4000000000LL;          // bound of the waits that drain a pass that timed out (clock64
                                                      // cycles; the pipeline's own take PassArgs::budget)
constexpr int F_TOP = 14;                             // W' < 2^TOP: TOP + SA + 1 bits fit ND_A signed bytes

template <int K, bool HESS> struct FDim {
    static constexpr int NV = HESS ? K * (K + 1) / 2 : K;    // sums per row
    static constexpr int NG = f64_groups(NV);                // column groups (grid.z)
    static constexpr int PER = (NV + NG - 1) / NG;           // sums per group
    static constexpr int NHP = (PER + 15) / 16 * 16;         // MMA columns of one order, zero beyond PER
    static constexpr int STR = f64_stride(PER);              // TMEM columns from one order to the next
    static constexpr int NPC = NHP / 4;                      // columns per order read out by one thread
    // with 16 columns per order, one MMA takes a weight digit with all product digits
    // (order d + b follows order d + b - 1 as the B rows do); orders from F_NORD on are
    // formed too, and not read
    static constexpr bool STACK = NHP == 16;
    static constexpr int COLS = STACK ? (F_NDA + F_NDB - 1) * 16 : (F_NORD - 1) * STR + NHP;
    static constexpr int TCOLS = COLS <= 256 ? 256 : 512;
    static constexpr int KS = (K + 1) | 1;                   // row stride (doubles): odd, so rows differ in banks;
                                                             // entry K of a row: its exponent
    static constexpr int B_TILE = F_NDB * NHP * F_KD * 2;
    static constexpr int ROWS = F_KD * KS * 8;
    static constexpr int IMG = NG * B_TILE + ROWS;           // image bytes per stage
    static constexpr int SLOT = ROWS + 512;                  // + 128 class words
};
constexpr int F_LBO_B = 128, F_SBO_B = 512;
template <bool PS> constexpr int f_lbo() { return PS ? 144 : 128; }   // P side: padded, so that a warp's
template <bool PS> constexpr int f_sbo() { return 4 * f_lbo<PS>(); }  // 32-bit stores hit distinct banks
template <bool PS> constexpr int f_atile() { return 16 * f_sbo<PS>(); }

struct FSync {
    uint64_t full[F_RING];    // vectors and class words landed
    uint64_t fullb[F_BRING];  // B tile landed
    uint64_t gen;        // the generator warps have written a stage's digits (one arrival per warp)
    uint64_t mma;        // a stage's MMAs are done
    uint32_t tslot;
    int bad, issued, loaded, loadedb;
};

template <int K, bool HESS, bool PS> constexpr size_t f_smem() {
    using D = FDim<K, HESS>;
    return 128 + (size_t)F_NDA * f_atile<PS>() + (size_t)F_BRING * D::B_TILE + (size_t)F_RING * D::SLOT + 128 * D::KS * 8 +
           F_GEN_WARPS * 256 * (8 + 2) + sizeof(FSync);
}

// Per block: whether it met an entry of Q or P outside [lo, 1] (bit patterns; an ulp or
// two above 1 passes, which a projection onto the simplex of one variable leaves).
// Block 0 also clears the flag of out-of-range weights.
__global__ void __launch_bounds__(256) k_f64_range(const double* __restrict__ q, int64_t nq,
                                                   const double* __restrict__ p, int64_t np, unsigned long long lo,
                                                   unsigned* __restrict__ off, int* __restrict__ flag) {
    const unsigned long long span = 0x3FF0000000000010ull - lo;
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x, stride = (int64_t)gridDim.x * 256;
    bool out = false;
    for (int64_t a = t; a < nq; a += stride) out |= (unsigned long long)__double_as_longlong(q[a]) - lo > span;
    for (int64_t a = t; a < np; a += stride) out |= (unsigned long long)__double_as_longlong(p[a]) - lo > span;
    const int any = __syncthreads_or(out);
    if (threadIdx.x == 0) off[blockIdx.x] = any ? 1u : 0u;
    if (t == 0) *flag = 0;
}

// The exponent kept with a row (entry K).
__device__ __forceinline__ int f64_row_exp(const double* row, int K) { return __double2loint(row[K]); }

// Fixed point of w 2^sh (w >= 0) in units of 2^-S, plus 128 in every one of the low
// BYTES bytes: byte d minus 128 is then the signed digit of weight 256^d.
template <int S, int BYTES>
__device__ __forceinline__ void f64_fix(double w, int sh, uint32_t (&x)[3]) {
    const uint32_t hi = (uint32_t)__double2hiint(w), lo = (uint32_t)__double2loint(w);
    const int e = (int)(hi >> 20) - 1023 + (S - 52) + sh;   // of the 53-bit integer m
    uint64_t m = ((uint64_t)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
    if (hi < 0x100000u) m = 0;                             // zero (no subnormals here)
    const int n = min(63, -e);
    const uint64_t l = e >= 0 ? m << (e & 63) : (m + (1ull << ((n - 1) & 63))) >> (n & 63);   // rounded
    const uint32_t h = e > 0 ? (uint32_t)(m >> ((64 - e) & 63)) : 0u;
    constexpr uint32_t OFF = BYTES >= 12 ? 0x80808080u : 0x80808080u >> (8 * (12 - BYTES));
    asm("add.cc.u32 %0, %3, %6;\n\t addc.cc.u32 %1, %4, %6;\n\t addc.u32 %2, %5, %7;"
        : "=&r"(x[0]), "=&r"(x[1]), "=&r"(x[2])
        : "r"((uint32_t)l), "r"((uint32_t)(l >> 32)), "r"(h), "r"(0x80808080u), "r"(OFF));
}

// Stage images: the digits of the products v_k v_k2 (or of v_k) of 32 reduction
// indices, in the shared-memory layout of the MMA's B operand, and the FP64
// vectors.  One warp per stage, lane = reduction index.  Indices past n get
// zeros (their class nibbles are padding).
// The index's exponent: of the sum of its entries (by_sum; a sum of 1 with a few ulps
// counts as 1), else of the largest.
template <int K, bool HESS>
__global__ void __launch_bounds__(128) k_f64_img(const double* __restrict__ v, int64_t n, int64_t stages, bool by_sum,
                                                 uint8_t* __restrict__ img) {
    using D = FDim<K, HESS>;
    const int lane = threadIdx.x & 31;
    const int64_t st = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (st >= stages) return;
    const int64_t a = st * F_KD + lane;
    uint8_t* base = img + st * D::IMG;
    double w[K], sum = 0.0;
    int mx = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        w[k] = a < n ? v[(int64_t)K * a + k] : 0.0;
        mx = max(mx, __double2hiint(w[k]));
        if (by_sum) sum += w[k];
    }
    const int f = mx ? f64_exponent(by_sum ? __double2hiint(sum) - 1 : mx) : 0;
    double* rows = reinterpret_cast<double*>(base + D::NG * D::B_TILE) + lane * D::KS;
#pragma unroll
    for (int k = 0; k < K; ++k) rows[k] = w[k];
    rows[K] = __longlong_as_double((long long)f);
    auto put = [&](int c, double y) {   // sum c, y 2^(-f or -2f) in [0, 1.01)
        const int g = c / D::PER, col = c - g * D::PER;
        uint32_t u[3];
        f64_fix<F_SB, F_NDB>(y, HESS ? -2 * f : -f, u);
        uint8_t* tile = base + g * D::B_TILE;
#pragma unroll
        for (int b = 0; b < F_NDB; ++b) {
            const int row = b * D::NHP + col, byte = F_NDB - 1 - b;
            const int d = (int)((u[byte >> 2] >> (8 * (byte & 3))) & 0xFF) - 128;
            uint16_t h;
            asm("cvt.rn.f16.s32 %0, %1;" : "=h"(h) : "r"(d));
            *reinterpret_cast<uint16_t*>(tile + (row >> 3) * F_SBO_B + (lane >> 3) * F_LBO_B + (row & 7) * 16 +
                                         (lane & 7) * 2) = h;
        }
    };
    if (HESS) {
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int k2 = k; k2 < K; ++k2) put(tri_idx<K>(k, k2), w[k] * w[k2]);
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) put(k, w[k]);
    }
    // padding columns are zero
    for (int g = 0; g < D::NG; ++g)
        for (int col = min(D::PER, D::NV - g * D::PER); col < D::NHP; ++col)
            for (int b = 0; b < F_NDB; ++b) {
                const int row = b * D::NHP + col;
                *reinterpret_cast<uint16_t*>(base + g * D::B_TILE + (row >> 3) * F_SBO_B + (lane >> 3) * F_LBO_B +
                                             (row & 7) * 16 + (lane & 7) * 2) = 0;
            }
}

__device__ __forceinline__ uint32_t f64_h2(uint32_t pair_bytes, uint32_t sel) {
    // two digit bytes -> packed FP16 integers: (1024 + byte) - 1152
    uint32_t h, d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(h) : "r"(pair_bytes), "r"(0x64646464u), "r"(sel));
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(h), "r"(0xE480E480u));
    return d;
}
// The four digits of word w of two elements: digit 4w + t in out[t].
__device__ __forceinline__ void f64_digits4(uint32_t x0, uint32_t x1, uint32_t (&out)[4]) {
    const uint32_t p01 = __byte_perm(x0, x1, 0x5140), p23 = __byte_perm(x0, x1, 0x7362);
    out[0] = f64_h2(p01, 0x4140);
    out[1] = f64_h2(p01, 0x4342);
    out[2] = f64_h2(p23, 0x4140);
    out[3] = f64_h2(p23, 0x4342);
}

// A wait of a whole warp: true if the phase is complete in time and no warp of the CTA
// has given up.  The lanes decide together, so that they leave together.
__device__ __forceinline__ bool f_wait(FSync* sy, uint64_t* bar, int phase, const PassArgs& a) {
    const bool ok = mbar_wait(bar, (uint32_t)(phase & 1), a.budget);
    if (!ok) {
        *(volatile int*)&sy->bad = 1;
        a.slots[S_TC_TIMEOUT] = 1.0;
    }
    return __all_sync(0xffffffffu, ok && *(volatile const int*)&sy->bad == 0);
}

// Weights of a warp's 2 x 32 pairs: lane = individual, blocks bb = 0, 1 of
// class nib[bb].  qrow: the 32 individuals' vectors; prow: the 8 columns'
// vectors (c = 4 bb + h).  The needed (pair, haplotype) items are listed by
// ballot and spread evenly over the lanes (4 rounds of 32 for 64 pairs instead
// of 8); then the pairs whose counts depend on qp, again listed, are finished
// from their reciprocals.  Results in rb[c][lane] (needed items only).
template <int K, bool HESS>
__device__ __forceinline__ void f64_weights(const unsigned (&nib)[2], const double* qrow, const double* prow,
                                            double* rb, uint16_t* list) {
    constexpr int KS = FDim<K, HESS>::KS;
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    int n = 0;
    unsigned need[2], cpl[2];
#pragma unroll
    for (int bb = 0; bb < 2; ++bb) {
        need[bb] = (unsigned)(TAB_NEED >> (4 * nib[bb])) & 0xFu;
        cpl[bb] = (TAB_CPLX >> nib[bb]) & 1u;
        const unsigned tag = lane | (__popc(need[bb]) == 1 ? 256u : 0u) | (cpl[bb] ? 512u : 0u);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const bool has = (need[bb] >> h) & 1u;
            const unsigned bal = __ballot_sync(0xffffffffu, has);
            if (has) list[n + __popc(bal & lt)] = (uint16_t)(tag | ((4 * bb + h) << 5));
            n += __popc(bal);
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const bool on = base + (int)lane < n;
        const unsigned it = on ? list[base + lane] : list[n - 1];
        const double* q = qrow + (it & 31u) * KS;
        const double* p = prow + ((it >> 5) & 7u) * KS;
        double s = q[0] * p[0];
#pragma unroll
        for (int k = 1; k < K; ++k) s = fma(q[k], p[k], s);
        const double r = rcp64(s);
        double w = r;                                   // left for the second part
        if (!(it & 512u)) {
            if (HESS) w = r * r;
            if (it & 256u) {                            // both copies: times 2, by the exponent where that is in range
                const unsigned ex = ((unsigned)__double2hiint(w) >> 20) & 0x7FFu;
                if (ex - 1u < 2045u) w = __hiloint2double(__double2hiint(w) + 0x00100000, __double2loint(w));
            }
        }
        if (on) rb[(it & 255u)] = w;                    // it & 255 = 32 c + lane
    }
    __syncwarp();
    // pairs with qp-dependent counts: a <-> b, c <-> d share a factor, with
    // x = r_a r_b, y = r_c r_d:
    //   het/het        (0,3,1,2): c_0 = c_3 = y/(x+y), c_1 = c_2 = x/(x+y)
    //   SNP 1 missing  (0,2,1,3), SNP 2 missing (0,1,2,3):
    //                  u = f r_a r_b / (r_a + r_b) = f / (qp_a + qp_b), f = copies in that set
    int nc = 0;
#pragma unroll
    for (int bb = 0; bb < 2; ++bb) {
        const unsigned bal = __ballot_sync(0xffffffffu, cpl[bb] != 0u);
        if (cpl[bb]) list[nc + __popc(bal & lt)] = (uint16_t)(lane | (nib[bb] << 6) | (bb << 5));
        nc += __popc(bal);
    }
    __syncwarp();
    // two lanes per pair, one for each set
#pragma unroll 1
    for (int base = 0; base < 2 * nc; base += 32) {
        const int slot = base + (int)lane;
        const unsigned it = list[min(slot >> 1, nc - 1)], set = lane & 1u;
        const unsigned nb = it >> 6, nd = (unsigned)(TAB_NEED >> (4 * nb)) & 0xFu;
        const bool hh = nb == NIB_HH, m1 = (nb & 3u) == 1u;
        const int ia = set ? (hh || m1 ? 1 : 2) : 0, ib = set ? (hh ? 2 : 3) : (hh ? 3 : (m1 ? 2 : 1));
        double* rp = rb + ((it >> 5) & 1u) * 128 + (it & 31u);
        const bool mine = slot < 2 * nc && ((nd >> ia) & 1u);    // a set is needed as a whole
        const bool both = __shfl_xor_sync(0xffffffffu, mine, 1) && mine;
        const double ra = mine ? rp[32 * ia] : 1.0, rbb = mine ? rp[32 * ib] : 1.0;
        const double own = ra * rbb, oth = __shfl_xor_sync(0xffffffffu, own, 1);
        const double e = (hh ? oth : own) * rcp64((hh ? own : ra) + (hh ? oth : rbb));
        const double f = both ? 1.0 : 2.0;
        const double ma = hh ? ra : f, mb = hh ? rbb : f;
        if (mine) {
            rp[32 * ia] = HESS ? (e * ra) * ma : e * ma;
            rp[32 * ib] = HESS ? (e * rbb) * mb : e * mb;
        }
    }
    __syncwarp();
}

// Whether w 2^sh is too large for the digits.
__device__ __forceinline__ bool f64_out_of_range(double w, int sh) {
    return (int)((uint32_t)__double2hiint(w) >> 20) + sh >= 1023 + F_TOP;
}

// A weight outside that range (see the top of the file), by a whole warp: its products
// with the index's vector, times 2^s, each below 2^38, in units of 2^-72, as three
// words of 37 bits, so that 2^26 of them fit the row's 64-bit integers.  The lanes take
// one product each, and all of it is integer work but the products themselves.
template <int K, bool HESS>
__device__ __noinline__ void f64_rare(double w, int s, const double* v, int c0, int c1, F64Rare ra, int64_t rows,
                                      int64_t row) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) atomicOr(ra.flag, 1);
    for (int c = c0 + lane; c < c1; c += 32) {
        int k = c, k2 = c;
        if (HESS) tri_pair<K>(c, k, k2);
        const unsigned long long y = (unsigned long long)__double_as_longlong(HESS ? w * (v[k] * v[k2]) : w * v[k]);
        const int e = (int)(y >> 52) - 1075 + 72 + s;
        const unsigned long long m = (y & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
        const unsigned __int128 x = e >= 0 ? (unsigned __int128)m << e
                                           : e > -54 ? (m + (1ull << (-e - 1))) >> -e : 0ull;
        constexpr unsigned long long M37 = (1ull << 37) - 1;
        unsigned long long* out = reinterpret_cast<unsigned long long*>(ra.i) + c * rows + row;
        const int64_t word = FDim<K, HESS>::NV * rows;
        atomicAdd(out, (unsigned long long)(x >> 74));
        atomicAdd(out + word, (unsigned long long)(x >> 37) & M37);
        atomicAdd(out + 2 * word, (unsigned long long)x & M37);
    }
    __syncwarp();
}

// ------------------------------------------------------------------ the pass
// PS = false (Q side): CTA rows = 128 individuals, stage = one word column (8
// blocks = 32 columns m); warp w: individuals 32 (w & 3) .. +31, blocks
// 2 (w >> 2), +1.  PS = true (P side): CTA rows = the 128 columns m of 32
// blocks, stage = 32 individuals; warp w: blocks 2w, 2w+1.  Chunks of the
// reduction along grid.y, column groups along grid.z.
// What bounds it: the FP64 unit, busy 74% of the clocks at K = 5 and 80% at K = 8 (K + 1
// operations per needed haplotype, 7 per pair with qp-dependent counts), then a warp's
// own chain from class to digits, in which the 16 warps move together; issue 42%.  One
// CTA per SM: a stage's FP64 work (registers and warp-private shared memory) runs while
// the MMAs of the stage before read the one set of digit tiles (two sets do not fit
// beside the warps' buffers).  Writing and issuing the digits in three words, so that a
// stage's first MMAs need not wait for its last digits, gained nothing.
// 10,000 individuals x 5,000 blocks, K = 5, Q pass: 3.43 ms with the reciprocals in FP64
// and 10 x 8 digits, 2.68 with integer reciprocals, 2.79 with 9 x 11 digits and an MMA per
// digit pair, 2.32 with one per weight digit; P pass 2.43.  50,000 x 4,000, K = 8, where
// every digit pair is an MMA of its own: 11.7 ms on either side.
template <int K, bool HESS, bool PS>
__global__ void __launch_bounds__(F_THREADS, 1) k_f64_pass(PassArgs a, F64Args fa) {
    using D = FDim<K, HESS>;
    constexpr int LBO = f_lbo<PS>(), SBO = f_sbo<PS>(), AT = f_atile<PS>();
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
    uint8_t* ring = smem + F_NDA * AT + F_BRING * D::B_TILE;
    double* fix = reinterpret_cast<double*>(ring + F_RING * D::SLOT);      // [128][KS]
    double* rbuf = fix + 128 * D::KS;                                      // [GEN_WARPS][8][32]
    uint16_t* lists = reinterpret_cast<uint16_t*>(rbuf + F_GEN_WARPS * 256);
    FSync* sy = reinterpret_cast<FSync*>(lists + F_GEN_WARPS * 256);
    const uint32_t sA = smem_u32(smem), sB = sA + F_NDA * AT, sR = smem_u32(ring);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int grp = blockIdx.z;
    const int64_t row0 = (int64_t)blockIdx.x * 128;
    // stages of this CTA
    const int64_t s0 = (int64_t)blockIdx.y * a.per_chunk;
    const int ns = (int)(min(fa.stages, s0 + a.per_chunk) - s0);
    const int nwc = PS ? (int)min((int64_t)4, (int64_t)a.JW - (int64_t)blockIdx.x * 4) : 1;

    // inputs that the general passes take (k_accum_q, k_accum_p)
    if (__syncthreads_or(tid < fa.noff && fa.off[tid] != 0u)) return;
    if (warp == F_GEN_WARPS) tmem_alloc<D::TCOLS>(&sy->tslot);
    if (tid == 0) {
        for (int r = 0; r < F_RING; ++r) mbar_init(&sy->full[r], 1);
        for (int r = 0; r < F_BRING; ++r) mbar_init(&sy->fullb[r], 1);
        mbar_init(&sy->gen, F_GEN_WARPS);
        mbar_init(&sy->mma, 1);
        sy->bad = 0;
        sy->issued = 0;
        sy->loaded = 0;
        sy->loadedb = 0;
        mbar_fence_init();
    }
    // the rows' own vectors
    const double* own = PS ? a.p : a.q;
    const int64_t nown = PS ? 4 * a.J : a.I;
    for (int t = tid; t < 128 * K; t += F_THREADS) {
        const int r = t / K, k = t - r * K;
        fix[r * D::KS + k] = row0 + r < nown ? own[(row0 + r) * K + k] : 0.25;
    }
    if (PS && HESS && tid < 128) {        // the rows' exponents
        int mx = 0;
#pragma unroll
        for (int k = 0; k < K; ++k)
            mx = max(mx, __double2hiint(row0 + tid < nown ? own[(row0 + tid) * K + k] : 0.25));
        fix[tid * D::KS + K] = __longlong_as_double((long long)f64_exponent(mx));
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, sy->tslot, 0);

    if (warp == F_GEN_WARPS) {
        const uint32_t el = elect_lane();
        auto copy = [&](uint32_t d, const void* g, uint32_t bytes, uint64_t* bar) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"(d), "l"(g), "r"(bytes), "r"(smem_u32(bar)) : "memory");
        };
        auto expect = [&](uint64_t* bar, uint32_t bytes) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
        };
        auto load_b = [&](int s) {
            uint64_t* bar = &sy->fullb[s % F_BRING];
            expect(bar, (uint32_t)D::B_TILE);
            copy(sB + (s % F_BRING) * D::B_TILE, a.img + (s0 + s) * D::IMG + grp * D::B_TILE, D::B_TILE, bar);
            *(volatile int*)&sy->loadedb = s + 1;
        };
        auto load = [&](int s) {          // vectors and class words
            const uint32_t dst = sR + (s % F_RING) * D::SLOT;
            uint64_t* bar = &sy->full[s % F_RING];
            expect(bar, (uint32_t)D::ROWS + (PS ? 128u * nwc : 512u));
            copy(dst, a.img + (s0 + s) * D::IMG + D::NG * D::B_TILE, D::ROWS, bar);
            if (PS) {
                for (int w = 0; w < nwc; ++w)
                    copy(dst + D::ROWS + 128 * w, a.G + ((int64_t)blockIdx.x * 4 + w) * a.Ipad + (s0 + s) * F_KD, 128,
                         bar);
            } else {
                copy(dst + D::ROWS, a.G + (s0 + s) * a.Ipad + row0, 512, bar);
            }
            *(volatile int*)&sy->loaded = s + 1;
        };
        if (el) {
            for (int s = 0; s < F_RING && s < ns; ++s) load(s);
            for (int s = 0; s < F_BRING && s < ns; ++s) load_b(s);
        }
        for (int s = 0; s < ns; ++s) {
            // all digits of the stage written, and every warp past stage s-1
            if (!f_wait(sy, &sy->gen, s, a)) break;
            // the slots of stage s-1: its MMAs are done (every warp waited for
            // them before it arrived for stage s) and its vectors are read
            if (el && s >= 1) {
                if (s + 2 < ns) load(s + 2);
                if (s + 1 < ns) load_b(s + 1);
            }
            if (!f_wait(sy, &sy->fullb[s % F_BRING], s / F_BRING, a)) break;
            fence_after();
            const uint64_t dA = sdesc(sA, LBO, SBO), dB = sdesc(sB + (s % F_BRING) * D::B_TILE, F_LBO_B, F_SBO_B);
            // One MMA per digit pair (or weight digit): all of one shape, so that they
            // execute in issue order where they share accumulators.  Where STR < NHP an
            // order's zero columns add 0 to the next order's first ones.
#pragma unroll 1
            for (int d = 0; d < F_NDA; ++d)
                if (D::STACK) {
#pragma unroll
                    for (int ks = 0; ks < F_KD / 16; ++ks)
                        mma_bf16(tmem + d * 16, dA + (uint64_t)((d * AT + ks * 2 * LBO) >> 4),
                                 dB + (uint64_t)((ks * 2 * F_LBO_B) >> 4), idesc_f16(F_NDB * 16), 1u, el);
                } else
#pragma unroll
                for (int b = 0; b < F_NDB; ++b) {
                    if (d + b >= F_NORD) break;
#pragma unroll
                    for (int ks = 0; ks < F_KD / 16; ++ks)
                        mma_bf16(tmem + (d + b) * D::STR, dA + (uint64_t)((d * AT + ks * 2 * LBO) >> 4),
                                 dB + (uint64_t)((b * (D::NHP / 8) * F_SBO_B + ks * 2 * F_LBO_B) >> 4),
                                 idesc_f16(D::NHP), 1u, el);
                }
            commit(&sy->mma, el);
            if (el) *(volatile int*)&sy->issued = s + 1;
        }
        __syncwarp();
    } else {
        constexpr int NPC = D::NPC;
        const int col0 = (warp >> 2) * NPC;                  // this thread's columns of an order
        const bool cols = col0 < D::STR;                     // (a quarter of the warps has none where STR < NHP)
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)col0;
        __int128 acc[NPC];                                   // units 2^-94, of order 12
#pragma unroll
        for (int c = 0; c < NPC; ++c) acc[c] = 0;
        // the window's columns go to the integer sums and are cleared
        auto zero_cols = [&]() {
            if (cols)
#pragma unroll
                for (int o = 0; o < F_NORD; ++o)
#pragma unroll
                    for (int c = 0; c < NPC; c += 4)
                        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};"
                                     :: "r"(tl + (uint32_t)(o * D::STR + c)), "r"(0u) : "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            fence_before();
        };
        // orders O0 .. O1 of four columns, Horner in base 256 (at most 2^24 each)
        auto read_orders = [&](int c, int o0, int o1, long long (&t)[4]) {
            uint32_t v[5][4];
#pragma unroll
            for (int o = 0; o < 5; ++o)
                if (o0 + o <= o1)
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(v[o][0]), "=r"(v[o][1]), "=r"(v[o][2]), "=r"(v[o][3])
                                 : "r"(tl + (uint32_t)((o0 + o) * D::STR + c)));
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                t[x] = 0;
#pragma unroll
                for (int o = 0; o < 5; ++o)
                    if (o0 + o <= o1) t[x] = t[x] * 256 + __float2int_rz(__uint_as_float(v[o][x]));
            }
        };
        auto read_out = [&]() {
            fence_after();
            if (cols)
#pragma unroll
                for (int c = 0; c < NPC; c += 4) {
                    long long t0[4], t1[4], t2[4];           // units 2^-30, 2^-62, 2^-94
                    read_orders(c, 0, 4, t0);
                    read_orders(c, 5, 8, t1);
                    read_orders(c, 9, 12, t2);
#pragma unroll
                    for (int x = 0; x < 4; ++x)
                        acc[c + x] += ((__int128)t0[x] << 64) + ((__int128)t1[x] << 32) + t2[x];
                }
        };
        zero_cols();
        const int lr = 32 * (warp & 3) + lane;                          // TMEM lane (row) of this thread
        double* rb = rbuf + warp * 256;
        uint16_t* list = lists + warp * 256;
        int s = 0;
        for (; s < ns; ++s) {
            const uint8_t* slot = ring + (s % F_RING) * D::SLOT;
            if (!f_wait(sy, &sy->full[s % F_RING], s / F_RING, a)) break;
            const double* srow = reinterpret_cast<const double*>(slot);
            const uint32_t* words = reinterpret_cast<const uint32_t*>(slot + D::ROWS);
            unsigned nib[2];
            const double *qrow, *prow;
            if (PS) {
                const int64_t j = (int64_t)blockIdx.x * 32 + 2 * warp;
                const uint32_t word = (warp >> 2) < nwc ? words[32 * (warp >> 2) + lane] : HX_PAD_WORD;
                const int bit = 8 * (warp & 3);
                nib[0] = j < a.J ? (word >> bit) & 0xFu : HX_PAD_NIBBLE;
                nib[1] = j + 1 < a.J ? (word >> (bit + 4)) & 0xFu : HX_PAD_NIBBLE;
                qrow = srow;
                prow = fix + 8 * warp * D::KS;
            } else {
                const uint32_t word = words[lr];
                const int bit = 8 * (warp >> 2);
                nib[0] = (word >> bit) & 0xFu;
                nib[1] = (word >> (bit + 4)) & 0xFu;
                qrow = fix + 32 * (warp & 3) * D::KS;
                prow = srow + 8 * (warp >> 2) * D::KS;
            }
            f64_weights<K, HESS>(nib, qrow, prow, rb, list);
            double W[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                W[c] = (unsigned)(TAB_NEED >> (4 * nib[c >> 2] + (c & 3))) & 1u ? rb[32 * c + lane] : 0.0;
            }
            // powers of two to scale by: the exponents of the reduction indices, and the
            // rows' on the P side
            auto fexp = [&](int c) { return f64_row_exp(PS ? qrow + lane * D::KS : prow + c * D::KS, K); };
            auto gexp = [&](int c) { return PS && HESS ? f64_row_exp(prow + c * D::KS, K) : 0; };
            auto sh = [&](int c) { return (HESS ? 2 : 1) * fexp(c) + gexp(c); };
            bool big = false;
#pragma unroll
            for (int c = 0; c < 8; ++c) big |= f64_out_of_range(W[c], sh(c));
            if (__any_sync(0xffffffffu, big)) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const bool mine = f64_out_of_range(W[c], sh(c));
                    unsigned left = __ballot_sync(0xffffffffu, mine);
                    while (left) {
                        const int l = __ffs(left) - 1;
                        left &= left - 1;
                        f64_rare<K, HESS>(__shfl_sync(0xffffffffu, W[c], l), gexp(c),
                                          PS ? qrow + l * D::KS : prow + c * D::KS, grp * D::PER,
                                          min(D::NV, (grp + 1) * D::PER), fa.rare, nown,
                                          PS ? row0 + 8 * warp + c : row0 + 32 * (warp & 3) + l);
                    }
                    if (mine) W[c] = 0.0;
                }
            }
            __syncwarp();
            // the digit tiles and the accumulators are free once stage s-1's MMAs are done
            if (s > 0) {
                if (!f_wait(sy, &sy->mma, s - 1, a)) break;
                if (s % F_WIN == 0) {
                    read_out();
                    zero_cols();
                }
            }
            if (PS) {
                // lane pairs (2t, 2t+1) share 32-bit words of two reduction
                // indices: the even lane stores block 0's rows, the odd one block 1's
                const bool odd = lane & 1;
                const int shm = (HESS ? 2 : 1) * fexp(0), sho = __shfl_xor_sync(0xffffffffu, shm, 1);
                uint32_t x0[4][3], x1[4][3];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const double mine = odd ? W[4 + h] : W[h];
                    const double other = __shfl_xor_sync(0xffffffffu, odd ? W[h] : W[4 + h], 1);
                    const int g = gexp((odd ? 4 : 0) + h);
                    f64_fix<F_SA, F_NDA>(odd ? other : mine, (odd ? sho : shm) + g, x0[h]);
                    f64_fix<F_SA, F_NDA>(odd ? mine : other, (odd ? shm : sho) + g, x1[h]);
                }
                const uint32_t at = sA + warp * SBO + (lane >> 3) * LBO + (odd ? 64 : 0) + (lane & 6) * 2;
#pragma unroll
                for (int w = 0; w < 3; ++w)
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t dg[4];
                        f64_digits4(x0[h][w], x1[h][w], dg);
#pragma unroll
                        for (int t = 0; t < (w < 2 ? 4 : F_NDA - 8); ++t)
                            asm volatile("st.shared.b32 [%0], %1;"
                                         :: "r"(at + (uint32_t)((F_NDA - 1 - (4 * w + t)) * AT + 16 * h)), "r"(dg[t])
                                         : "memory");
                    }
            } else {
                uint32_t x[8][3];
#pragma unroll
                for (int c = 0; c < 8; ++c) f64_fix<F_SA, F_NDA>(W[c], sh(c), x[c]);
                const uint32_t at = sA + (lr >> 3) * SBO + (warp >> 2) * LBO + (lr & 7) * 16;
#pragma unroll
                for (int w = 0; w < 3; ++w) {
                    uint32_t dg[4][4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) f64_digits4(x[2 * e][w], x[2 * e + 1][w], dg[e]);
#pragma unroll
                    for (int t = 0; t < (w < 2 ? 4 : F_NDA - 8); ++t)
                        sts128(at + (uint32_t)((F_NDA - 1 - (4 * w + t)) * AT), dg[0][t], dg[1][t], dg[2][t], dg[3][t]);
                }
            }
            fence_async_smem();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sy->gen);
        }
        if (s == ns && ns > 0 && f_wait(sy, &sy->mma, ns - 1, a)) read_out();
        const int64_t rows = PS ? 4 * a.J : a.Ipad;
        const int64_t row = row0 + lr;
        if (row < rows) {
            double* out = a.part + (int64_t)blockIdx.y * D::NV * rows;
#pragma unroll
            for (int c = 0; c < NPC; ++c) {
                const int col = col0 + c;
                const int v = grp * D::PER + col;
                if (col < D::PER && v < D::NV)
                    out[(int64_t)v * rows + row] = scalbn((double)(long long)(acc[c] >> 64), -30) +
                                                   scalbn((double)(unsigned long long)acc[c], -94);
            }
        }
    }
    __syncthreads();
    if (sy->bad) {
        // a wait ran out: let the MMAs and copies that were issued end before
        // tensor and shared memory are released
        const int n = sy->issued, l = sy->loaded;
        if (n > 0) mbar_wait(&sy->mma, (uint32_t)((n - 1) & 1), F_BUDGET);
        for (int t = (l >= F_RING ? l - F_RING : 0); t < l; ++t)
            mbar_wait(&sy->full[t % F_RING], (uint32_t)((t / F_RING) & 1), F_BUDGET);
        const int lb = sy->loadedb;
        for (int t = (lb >= F_BRING ? lb - F_BRING : 0); t < lb; ++t)
            mbar_wait(&sy->fullb[t % F_BRING], (uint32_t)((t / F_BRING) & 1), F_BUDGET);
        __syncthreads();
    }
    fence_before();
    __syncthreads();
    if (warp == F_GEN_WARPS) {
        fence_after();
        tmem_dealloc<D::TCOLS>(tmem);
    }
}

}  // namespace
}  // namespace hx
