// hx_items.cuh -- which haplotypes of a pair a plain-method (FP64) pass has to
// evaluate.  GB300's FP64 unit is 1/64 as wide as its FP32 units, so those
// passes list the needed (individual, haplotype) items of a warp's pairs and
// spread them evenly over its lanes, instead of evaluating all four
// haplotypes of every pair.
#pragma once
#include "hx_common.cuh"

namespace hx {

// Needed haplotypes of a class (all four for the double heterozygote, none for
// double missing).
__host__ __device__ constexpr unsigned class_need(unsigned nib) {
    return nib == NIB_HH ? 0xFu : (class_m1(nib) | class_m2(nib));
}
__host__ __device__ constexpr uint64_t make_need() {
    uint64_t t = 0;
    for (unsigned n = 0; n < 16; ++n) t |= (uint64_t)class_need(n) << (4 * n);
    return t;
}
constexpr uint64_t TAB_NEED = make_need();
// Classes whose counts depend on qp: the double heterozygote and one SNP missing.
__host__ __device__ constexpr unsigned make_cplx() {
    unsigned t = 0;
    for (unsigned n = 0; n < 16; ++n)
        if (n == NIB_HH || ((((n & 3u) == 1u) != ((n >> 2) == 1u)))) t |= 1u << n;
    return t;
}
constexpr unsigned TAB_CPLX = make_cplx();

}  // namespace hx
