// Poseidon2 width 8 over Goldilocks for the host (the permutation of gl_poseidon2.cuh; same function, same tables).
//
// The device form counts 32-bit instructions; a host core has a 64 x 64 -> 128 multiplier, 128-bit adds in two
// instructions and out-of-order issue, so this form multiplies through unsigned __int128, keeps the linear layers
// as 128-bit sums with one reduction per output, and lets the S-box chain of an internal round overlap the other
// lanes' products. A round loop's host side (transcript, tree tops) is a chain of these permutations between two
// kernel launches, so their latency is on every proof's critical path.
#pragma once
#include <cstdint>
#include "../gl_poseidon2.cuh"
#include "host_field.hpp"

namespace mbhost {
namespace p2host {

using hf::u128;
constexpr uint64_t EPS = hf::GL_EPS;
static MB_HOT uint64_t red(u128 x) { return hf::gl_red(x); }   // any 128-bit value, loose result
static MB_HOT uint64_t mul(uint64_t a, uint64_t b) { return red((u128)a * b); }
static MB_HOT uint64_t sbox7(uint64_t x) {
    const uint64_t x2 = mul(x, x), x4 = mul(x2, x2), x3 = mul(x2, x);
    return mul(x4, x3);
}

// y = M4 x for M4 = [2 3 1 1; 1 2 3 1; 1 1 2 3; 3 1 1 2], as 128-bit sums (inputs below 2^64: outputs below 7 2^64).
static MB_HOT void mat4(const uint64_t* x, u128* y) {
    const u128 t01 = (u128)x[0] + x[1], t23 = (u128)x[2] + x[3];
    const u128 t0123 = t01 + t23;
    const u128 t01123 = t0123 + x[1], t01233 = t0123 + x[3];
    y[3] = t01233 + ((u128)x[0] << 1);
    y[1] = t01123 + ((u128)x[2] << 1);
    y[0] = t01123 + t01;
    y[2] = t01233 + t23;
}

// s <- [[2 M4, M4], [M4, 2 M4]] s + rc (rc may be null): sums stay below 22 2^64.
static MB_HOT void external_linear(uint64_t* s, const uint64_t* rc) {
    u128 a[4], b[4];
    mat4(s, a);
    mat4(s + 4, b);
    for (int i = 0; i < 4; i++) {
        const u128 sum = a[i] + b[i];
        s[i] = red(a[i] + sum + (rc ? rc[i] : 0));
        s[i + 4] = red(b[i] + sum + (rc ? rc[i + 4] : 0));
    }
}

// In place, for any host core.
static inline void permute_portable(uint64_t* s) {
    const uint64_t(*rc_ext)[8] = gl::h_p2_rc_ext;
    const uint64_t* rc_int = gl::h_p2_rc_int;
    const uint64_t* diag = gl::h_p2_diag;
    for (int i = 0; i < 8; i++) s[i] = red((u128)s[i] + rc_ext[0][i]);
    for (int r = 0; r < 4; r++) {
        for (int i = 0; i < 8; i++) s[i] = sbox7(s[i]);
        external_linear(s, r < 3 ? rc_ext[r + 1] : nullptr);
    }
    // Internal rounds: s_0 <- sbox(s_0 + rc), then s_i <- d_i s_i + sum_j s_j. The chain that matters is lane 0's:
    // with rest = the other lanes' sum (reduced beside the S-box), the new lane 0 is s0 (d_0 + 1) + rest + the next
    // round's constant in one 128-bit sum ((2^64 - 1) p + 2 (2^64 - 1) < 2^128), so a round costs the S-box and one
    // multiply-reduce on the chain.
    s[0] = red((u128)s[0] + rc_int[0]);
    const uint64_t d0p1 = diag[0] + 1;
    for (int r = 0; r < 22; r++) {
        u128 rest128 = 0;
        for (int i = 1; i < 8; i++) rest128 += s[i];
        const uint64_t rest = red(rest128);
        u128 prod[8];
        for (int i = 1; i < 8; i++) prod[i] = (u128)s[i] * diag[i] + rest;
        const uint64_t s0 = sbox7(s[0]);
        s[0] = red((u128)s0 * d0p1 + rest + (r < 21 ? rc_int[r + 1] : 0));
        for (int i = 1; i < 8; i++) s[i] = red(prod[i] + s0);
    }
    for (int i = 0; i < 8; i++) s[i] = red((u128)s[i] + rc_ext[4][i]);
    for (int r = 4; r < 8; r++) {
        for (int i = 0; i < 8; i++) s[i] = sbox7(s[i]);
        external_linear(s, r < 7 ? rc_ext[r + 1] : nullptr);
    }
    for (int i = 0; i < 8; i++) s[i] = s[i] >= gl::P ? s[i] - gl::P : s[i];
}

#if defined(__x86_64__)
// The same permutation for an x86-64 core with BMI2, the products and reductions in assembly. The compiled form above
// is bound by its micro-operations (about 14 per product and reduction, and the spills between them); here a product
// and its reduction are nine: the borrow of lo - hi_hi is a jump that is taken once in 2^32 products, hi_lo (2^32 - 1)
// is one multiplication, and only the last carry (a coin flip) is repaired without a branch. 0.85 -> 0.57 us a
// permutation on a 16-core Sapphire-Rapids-class host. In the internal rounds (d_0 + 1) x x^2 is formed beside x^3 and x^4, so that lane 0's
// next value is three products after this one instead of four, and the other lanes' sum is one round behind it.
#define MB_P2_RED                                                                                                     \
    "mov %k[hi], %k[t]\n\timul %[eps], %[t]\n\tshr $32, %[hi]\n\tsub %[hi], %[lo]\n\tjb 2f\n1:\tadd %[t], %[lo]\n\t"  \
    "sbb %k[t], %k[t]\n\tadd %[t], %[lo]\n\t.subsection 1\n2:\tsub %[eps], %[lo]\n\tjmp 1b\n\t.previous"
namespace bmi2 {
// a b, a b + c and a b + c + d mod p, loose ((2^64 - 1)^2 + 2 (2^64 - 1) < 2^128)
static MB_HOT uint64_t mul(uint64_t a, uint64_t b) {
    uint64_t lo, hi, t;
    asm("mulx %[b], %[lo], %[hi]\n\t" MB_P2_RED
        : [lo] "=&r"(lo), [hi] "=&r"(hi), [t] "=&r"(t) : [eps] "r"(EPS), "d"(a), [b] "rm"(b) : "cc");
    return lo;
}
static MB_HOT uint64_t mul_add(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t lo, hi, t;
    asm("mulx %[b], %[lo], %[hi]\n\tadd %[c], %[lo]\n\tadc $0, %[hi]\n\t" MB_P2_RED
        : [lo] "=&r"(lo), [hi] "=&r"(hi), [t] "=&r"(t) : [eps] "r"(EPS), "d"(a), [b] "rm"(b), [c] "r"(c) : "cc");
    return lo;
}
static MB_HOT uint64_t mul_add2(uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
    uint64_t lo, hi, t;
    asm("mulx %[b], %[lo], %[hi]\n\tadd %[c], %[lo]\n\tadc $0, %[hi]\n\tadd %[d], %[lo]\n\tadc $0, %[hi]\n\t" MB_P2_RED
        : [lo] "=&r"(lo), [hi] "=&r"(hi), [t] "=&r"(t)
        : [eps] "r"(EPS), "d"(a), [b] "rm"(b), [c] "r"(c), [d] "rm"(d) : "cc");
    return lo;
}
// hi 2^64 + lo mod p, loose, for hi < 2^32 (the wrapped sum is below hi EPS, so the repair cannot carry)
static MB_HOT uint64_t red_small(uint64_t lo, uint64_t hi) {
    uint64_t u = (hi << 32) - hi;
    asm("add %[u], %[lo]\n\tsbb %k[u], %k[u]\n\tadd %[u], %[lo]" : [lo] "+r"(lo), [u] "+r"(u) : : "cc");
    return lo;
}
static MB_HOT uint64_t red_small(u128 x) { return red_small((uint64_t)x, (uint64_t)(x >> 64)); }
static MB_HOT uint64_t sbox7(uint64_t x) {
    const uint64_t x2 = mul(x, x), x4 = mul(x2, x2), x3 = mul(x2, x);
    return mul(x4, x3);
}
static MB_HOT void full_round(uint64_t* s, const uint64_t* rc) {   // rc: the next round's constants
    s[0] = sbox7(s[0]); s[1] = sbox7(s[1]); s[2] = sbox7(s[2]); s[3] = sbox7(s[3]);   // unrolled by hand
    s[4] = sbox7(s[4]); s[5] = sbox7(s[5]); s[6] = sbox7(s[6]); s[7] = sbox7(s[7]);
    u128 a[4], b[4];
    mat4(s, a);
    mat4(s + 4, b);
    const auto out = [&](int i) __attribute__((always_inline)) {
        const u128 sum = a[i] + b[i];
        s[i] = red_small(a[i] + sum + rc[i]);
        s[i + 4] = red_small(b[i] + sum + rc[i + 4]);
    };
    out(0); out(1); out(2); out(3);
}
// A function of its own, on a 64-byte boundary: 580 ns wherever the linker puts a translation unit, 591 inlined and 585 unaligned (on
// the B200 machine's Xeon; on another Xeon, of 2.7 GHz, the three are within its noise, 765 ns).
__attribute__((noinline, aligned(64))) static void permute(uint64_t* st) {
    const uint64_t(*rc_ext)[8] = gl::h_p2_rc_ext;
    const uint64_t *rc_int = gl::h_p2_rc_int, *diag = gl::h_p2_diag;
    static const uint64_t none[8] = {};
    uint64_t s[8];
    for (int i = 0; i < 8; i++) s[i] = red_small((u128)st[i] + rc_ext[0][i]);
    for (int r = 0; r < 4; r++) full_round(s, r < 3 ? rc_ext[r + 1] : none);
    const uint64_t d0p1 = diag[0] + 1;
    uint64_t x = red_small((u128)s[0] + rc_int[0]);
    u128 sum = 0;
    for (int i = 1; i < 8; i++) sum += s[i];
    uint64_t rest = red_small(sum);   // sum of lanes 1 .. 7
    for (int r = 0; r < 22; r++) {
        const uint64_t x2 = mul(x, x), w = mul(x, d0p1), x4 = mul(x2, x2), w3 = mul(w, x2), x3 = mul(x2, x);
        x = mul_add2(x4, w3, rest, r < 21 ? rc_int[r + 1] : 0);
        const uint64_t all = red_small((u128)mul(x3, x4) + rest);
        uint64_t lo = 0, hi = 0;
        const auto lane = [&](int i) __attribute__((always_inline)) {
            const uint64_t v = s[i] = mul_add(s[i], diag[i], all);
            asm("add %[v], %[lo]\n\tadc $0, %[hi]" : [lo] "+r"(lo), [hi] "+r"(hi) : [v] "r"(v) : "cc");
        };
        lane(1); lane(2); lane(3); lane(4); lane(5); lane(6); lane(7);
        rest = red_small(lo, hi);
    }
    s[0] = x;
    for (int i = 0; i < 8; i++) s[i] = red_small((u128)s[i] + rc_ext[4][i]);
    for (int r = 4; r < 8; r++) full_round(s, r < 7 ? rc_ext[r + 1] : none);
    for (int i = 0; i < 8; i++) st[i] = s[i] >= gl::P ? s[i] - gl::P : s[i];
}
}  // namespace bmi2
#undef MB_P2_RED
static const bool have_bmi2 = [] { __builtin_cpu_init(); return __builtin_cpu_supports("bmi2") != 0; }();
#endif

// In place; any 64-bit words in, canonical residues out.
static inline void permute(uint64_t* s) {
#if defined(__x86_64__)
    if (have_bmi2) return bmi2::permute(s);
#endif
    permute_portable(s);
}

}  // namespace p2host
}  // namespace mbhost
