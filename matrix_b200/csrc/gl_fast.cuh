// Goldilocks arithmetic for kernels that run many permutations and can run one again: products and sums without their rare
// repairs, which are told of instead, and linear maps by small whole numbers on the FP64 pipe, which integer code leaves idle.
#pragma once
#include "gl_field.cuh"

#ifdef __CUDACC__
namespace gl {
namespace fast {
// Repairs left out so far. A borrow left as it is shows in the word it leaves: a high word of at least 2^32 - 1 - z4 (below). So
// the largest high word tells of them all, and of z4 + 1 right words in 2^32; a maximum goes to the other pipe than a carry kept in
// a register, and the same holds for an addition to which its own carry is added at once: 27.1 -> 23.4 cycles a product. Carries
// left out are counted.
struct Missed {
    uint32_t top, carries;
    // most: the largest z4 of the reductions so far. What is told of for nothing costs a whole exact permutation: with 63 here, a layer of
    // 2^14 permutations took 39 us instead of 23 one time in eight.
    __device__ __forceinline__ bool any(uint32_t most = 0) const { return top >= 0xFFFFFFFFu - most || carries != 0; }
};
// reduce_limbs without the repair; z4 2^128 = -z4 2^32. (A : z0) - (B1 : B0) borrows if A is less than B1 or B1 + 1, and B1 is z4 or, with
// A at least 1 then, z4 + 1: the high word comes out at 2^32 - 1 - z4 or above. Likewise in a sum (z4 = 0).
__device__ __forceinline__ uint64_t reduce(uint32_t z0, uint32_t z1, uint32_t z2, uint32_t z3, uint32_t z4, Missed& missed) {
    uint32_t A, B0, B1, r0, r1;
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %3, %4;\n\taddc.u32 %0, t, 0;\n\taddc.cc.u32 %1, %4, %5;\n\taddc.u32 %2, %6, 0;\n\t}"
        : "=&r"(A), "=&r"(B0), "=r"(B1) : "r"(z1), "r"(z2), "r"(z3), "r"(z4));
    asm("sub.cc.u32 %0, %2, %3;\n\tsubc.u32 %1, %4, %5;" : "=&r"(r0), "=r"(r1) : "r"(z0), "r"(B0), "r"(A), "r"(B1));
    missed.top = max(missed.top, r1);
    return pack64(r0, r1);
}
__device__ __forceinline__ uint64_t reduce(unsigned __int128 f, Missed& missed) {
    const uint64_t lo = (uint64_t)f, hi = (uint64_t)(f >> 64);
    return reduce(lo32(lo), hi32(lo), lo32(hi), hi32(hi), 0, missed);
}
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b, Missed& missed) { return reduce((unsigned __int128)a * b, missed); }
__device__ __forceinline__ uint64_t mul_add(uint64_t a, uint64_t b, uint64_t c, Missed& missed) {
    return reduce((unsigned __int128)a * b + c, missed);
}
// For code that waits for single results: a product less (the cross one doubled) takes 9 cycles off an S-box; where many run at a time,
// the shifts cost more than the product.
__device__ __forceinline__ uint64_t sqr(uint64_t a, Missed& missed) {
    const uint32_t a0 = lo32(a), a1 = hi32(a);
    const uint64_t e = (uint64_t)a0 * a0, f = (uint64_t)a1 * a1, o = (uint64_t)a0 * a1;
    uint32_t z1 = hi32(e), z2 = lo32(f), z3 = hi32(f);
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(z1), "+r"(z2), "+r"(z3) : "r"(lo32(o) << 1), "r"((uint32_t)(o >> 31)), "r"(hi32(o) >> 31));
    return reduce(lo32(e), z1, z2, z3, 0, missed);
}
// sums of words: 96 bits
struct Sum {
    uint32_t a, b, c;
};
// (b:a) + c EPS for c < 2^10; a carry out of b + c and a borrow of (b + c : a) - c are not repaired
__device__ __forceinline__ uint64_t reduce(Sum x, Missed& missed) {
    uint32_t r0, r1;
    asm("add.cc.u32 %1, %4, %5;\n\taddc.u32 %2, %2, 0;\n\tsub.cc.u32 %0, %3, %5;\n\tsubc.u32 %1, %1, 0;"
        : "=&r"(r0), "=&r"(r1), "+r"(missed.carries) : "r"(x.a), "r"(x.b), "r"(x.c));
    missed.top = max(missed.top, r1);
    return pack64(r0, r1);
}
// ---- whole numbers in doubles ------------------------------------------------------------------
// 2^52 + x is the word FP_ONE in front of x; sums of 32-bit halves with small weights stay far below 2^52, so every operation is
// exact, and the sum lies in the low words of 2^52 + sum again.
constexpr uint32_t FP_ONE = 0x43300000u;   // high word of 2^52
constexpr double TWO_52 = 4503599627370496.0;
__device__ __forceinline__ double whole(uint32_t x) { return __hiloint2double((int)FP_ONE, (int)x); }
// L + H 2^32 from LOW_HALF + L and HIGH_HALF + H, L and H < 2^42: FP_ONE in the high word of the first meets its complement in the low
// word of the second.
constexpr double LOW_HALF = TWO_52, HIGH_HALF = TWO_52 + (4294967296.0 - (double)FP_ONE);
__device__ __forceinline__ uint64_t from_halves(double l, double h, Missed& missed) {
    Sum x;
    x.a = (uint32_t)__double2loint(l);
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;"
        : "=&r"(x.b), "=r"(x.c)
        : "r"((uint32_t)__double2hiint(l)), "r"((uint32_t)__double2loint(h)), "r"((uint32_t)__double2hiint(h)), "n"(0u - FP_ONE - 1));
    return reduce(x, missed);
}

}  // namespace fast
}  // namespace gl
#endif
