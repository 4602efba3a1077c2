// The Monolith permutation (width 12) of both fields on a core with AVX-512 IFMA: the portable forms in
// agl_transcript.hpp and gl_monolith_host.hpp, twelve words at a time.
//
// A permutation between two kernel launches is a chain of layers, so its latency counts. Compiled for scalar
// registers a layer is about 800 micro-operations; here it is about 110 vector instructions:
//   * the state's 32-bit halves stay apart from the squares to the end of the next linear layer: a square is added
//     to its neighbour as two limb sums L + 2^32 H below 2^39, the circulant multiplies them by its small integers
//     (52-bit multiply-add, row sum 160: below 2^47), and one reduction per word and layer is left;
//   * the circulant is a sum over the twelve words: the pair (L_j, H_j) is broadcast from memory and multiplied by
//     column j, three vectors of four words each, in two chains.
// 0.49 -> 0.2 us a permutation on a Sapphire-Rapids-class host (0.73 -> 0.28 us on a 2.5 GHz Rocket Lake core).
#pragma once
#include <cstdint>
#if defined(__x86_64__)
#include <immintrin.h>

namespace mbhost {
namespace mono512 {

#define MB_AVX512 __attribute__((target("avx512f,avx512dq,avx512vl,avx512bw,avx512ifma")))
#define MB_AVX512_INLINE static inline __attribute__((always_inline)) MB_AVX512

static const bool available = [] {
    __builtin_cpu_init();
    return __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512dq") && __builtin_cpu_supports("avx512vl") &&
           __builtin_cpu_supports("avx512bw") && __builtin_cpu_supports("avx512ifma");
}();

// column j of the MDS circulant for the accumulator of words 4a .. 4a + 3, every entry twice (low, high half)
struct alignas(64) Columns {
    uint64_t c[12][3][8];
    constexpr Columns() : c() {
        constexpr int C[12] = {7, 23, 8, 26, 13, 10, 9, 7, 6, 22, 21, 8};
        for (int j = 0; j < 12; j++)
            for (int i = 0; i < 12; i++) { c[j][i / 4][2 * (i % 4)] = C[(j - i + 12) % 12]; c[j][i / 4][2 * (i % 4) + 1] = C[(j - i + 12) % 12]; }
    }
};
static constexpr Columns columns;

struct Agl {
    static constexpr uint64_t P = 0xFFFFFFFEFFFFFFE1ULL, C = 0x10000001FULL;
    // hi 2^64 mod p for hi below 2^16
    MB_AVX512_INLINE __m512i top(__m512i hi) { return _mm512_madd52lo_epu64(_mm512_setzero_si512(), hi, _mm512_set1_epi64(C)); }
    // x^2 from b = x_0^2, a = x_0 x_1, c = x_1^2 as limb sums (2^64 = 2^32 + 31, 2^96 = 32 2^32 + 31)
    MB_AVX512_INLINE void square(__m512i b, __m512i a, __m512i c, __m512i& L, __m512i& H) {
        const __m512i m = _mm512_set1_epi64(0xFFFFFFFFLL);
        const __m512i a1 = _mm512_srli_epi64(a, 32), a0 = _mm512_and_si512(a, m), c1 = _mm512_srli_epi64(c, 32), c0 = _mm512_and_si512(c, m);
        const __m512i z2 = _mm512_add_epi64(_mm512_add_epi64(a1, a1), c0);
        L = _mm512_madd52lo_epu64(_mm512_and_si512(b, m), _mm512_add_epi64(z2, c1), _mm512_set1_epi64(31));
        H = _mm512_add_epi64(_mm512_add_epi64(_mm512_srli_epi64(b, 32), _mm512_add_epi64(a0, a0)), _mm512_add_epi64(z2, _mm512_slli_epi64(c1, 5)));
    }
};
struct Gl {
    static constexpr uint64_t P = 0xFFFFFFFF00000001ULL, C = 0xFFFFFFFFULL;
    MB_AVX512_INLINE __m512i top(__m512i hi) { return _mm512_sub_epi64(_mm512_slli_epi64(hi, 32), hi); }
    MB_AVX512_INLINE void square(__m512i b, __m512i a, __m512i c, __m512i& L, __m512i& H) {
        const __m512i m = _mm512_set1_epi64(0xFFFFFFFFLL);
        const __m512i a1 = _mm512_srli_epi64(a, 32), a0 = _mm512_and_si512(a, m), c1 = _mm512_srli_epi64(c, 32), c0 = _mm512_and_si512(c, m);
        const __m512i z2 = _mm512_add_epi64(_mm512_add_epi64(a1, a1), c0);
        // 2^64 = 2^32 - 1, 2^96 = -1; 16 p split as (16 2^32 + 16) + 2^32 (16 2^32 - 32) keeps both sums positive
        L = _mm512_sub_epi64(_mm512_add_epi64(_mm512_and_si512(b, m), _mm512_set1_epi64(16 * 0x100000000LL + 16)), _mm512_add_epi64(z2, c1));
        H = _mm512_add_epi64(_mm512_add_epi64(_mm512_srli_epi64(b, 32), _mm512_add_epi64(a0, a0)), _mm512_add_epi64(z2, _mm512_set1_epi64(16 * 0x100000000LL - 32)));
    }
};
// L + 2^32 H mod p, loose, for L, H below 2^48 (the wrapped sum is below hi C < 2^50: one repair)
template <class F> MB_AVX512_INLINE __m512i reduce(__m512i L, __m512i H) {
    const __m512i s = _mm512_add_epi64(L, _mm512_slli_epi64(H, 32));
    const __mmask8 k = _mm512_cmplt_epu64_mask(s, L);
    const __m512i h = _mm512_srli_epi64(H, 32);
    const __m512i hi = _mm512_mask_sub_epi64(h, k, h, _mm512_set1_epi64(-1));
    const __m512i t = F::top(hi), r = _mm512_add_epi64(s, t);
    return _mm512_mask_add_epi64(r, _mm512_cmplt_epu64_mask(r, t), r, _mm512_set1_epi64(F::C));
}
MB_AVX512_INLINE __m512i rotl8(__m512i x, int k, uint8_t low) {   // every byte rotated left by k; low: mask of the k low bits
    const __m512i m = _mm512_set1_epi8((char)low);
    return _mm512_ternarylogic_epi64(m, _mm512_srli_epi64(x, 8 - k), _mm512_slli_epi64(x, k), 0xCA);
}
MB_AVX512_INLINE __m512i bar(__m512i x) {
    const __m512i l1 = rotl8(x, 1, 1), l2 = rotl8(x, 2, 3), l3 = rotl8(x, 3, 7);
    const __m512i a = _mm512_ternarylogic_epi64(l1, l2, l3, 0x08);   // ~l1 & l2 & l3
    return rotl8(_mm512_xor_si512(x, a), 1, 1);
}
// In place; any 64-bit words in, canonical residues out. rc[0 .. 6]: the constants of the seven linear layers.
template <class F> MB_AVX512 static void permute(uint64_t* st, const uint64_t (*rc)[12]) {
    alignas(64) uint64_t buf[24];
    const __m512i m32 = _mm512_set1_epi64(0xFFFFFFFFLL);
    // halves of word i at buf[2 i], buf[2 i + 1]
    for (int i = 0; i < 12; i++) { buf[2 * i] = (uint32_t)st[i]; buf[2 * i + 1] = st[i] >> 32; }
    __m512i A, B;   // words 0 4 1 5 2 6 3 7 and 8 8 9 9 10 10 11 11
    for (int r = 0;; r++) {
        __m512i acc[3], acd[3];
        for (int a = 0; a < 3; a++) {
            // the round constants' halves: 64-bit words spread as (low, high)
            const __m256i w = _mm256_loadu_si256((const __m256i*)(rc[r] + 4 * a));
            acc[a] = _mm512_cvtepu32_epi64(w);
            acd[a] = _mm512_setzero_si512();
        }
        for (int j = 0; j < 12; j += 2) {
            const __m512i x = _mm512_broadcast_i64x2(_mm_load_si128((const __m128i*)(buf + 2 * j)));
            const __m512i y = _mm512_broadcast_i64x2(_mm_load_si128((const __m128i*)(buf + 2 * j + 2)));
            for (int a = 0; a < 3; a++) {
                acc[a] = _mm512_madd52lo_epu64(acc[a], x, _mm512_load_si512(columns.c[j][a]));
                acd[a] = _mm512_madd52lo_epu64(acd[a], y, _mm512_load_si512(columns.c[j + 1][a]));
            }
        }
        for (int a = 0; a < 3; a++) acc[a] = _mm512_add_epi64(acc[a], acd[a]);
        A = reduce<F>(_mm512_unpacklo_epi64(acc[0], acc[1]), _mm512_unpackhi_epi64(acc[0], acc[1]));
        B = reduce<F>(_mm512_unpacklo_epi64(acc[2], acc[2]), _mm512_unpackhi_epi64(acc[2], acc[2]));
        if (r == 6) break;
        // bars on words 0 .. 3 (lanes 0 2 4 6 of A), canonical
        const __m512i p = _mm512_set1_epi64((long long)F::P);
        const __m512i Ac = _mm512_mask_sub_epi64(A, _mm512_cmpge_epu64_mask(A, p), A, p);
        A = _mm512_mask_mov_epi64(A, 0x55, bar(Ac));
        const __m512i Ah = _mm512_srli_epi64(A, 32), Bh = _mm512_srli_epi64(B, 32);
        __m512i LA, HA, LB, HB;
        F::square(_mm512_mul_epu32(A, A), _mm512_mul_epu32(A, Ah), _mm512_mul_epu32(Ah, Ah), LA, HA);
        F::square(_mm512_mul_epu32(B, B), _mm512_mul_epu32(B, Bh), _mm512_mul_epu32(Bh, Bh), LB, HB);
        // s_i += (word before)^2: the squares' halves move up one word
        const __m512i ia = _mm512_setr_epi64(0, 6, 0, 1, 2, 3, 4, 5), ib = _mm512_setr_epi64(7, 7, 8, 8, 10, 10, 12, 12);
        const __m512i lb = _mm512_permutex2var_epi64(LA, ib, LB), hb = _mm512_permutex2var_epi64(HA, ib, HB);
        LA = _mm512_add_epi64(_mm512_maskz_permutexvar_epi64(0xFE, ia, LA), _mm512_and_si512(A, m32));
        HA = _mm512_add_epi64(_mm512_maskz_permutexvar_epi64(0xFE, ia, HA), Ah);
        LB = _mm512_add_epi64(lb, _mm512_and_si512(B, m32));
        HB = _mm512_add_epi64(hb, Bh);
        _mm512_store_si512(buf, _mm512_unpacklo_epi64(LA, HA));
        _mm512_store_si512(buf + 8, _mm512_unpackhi_epi64(LA, HA));
        _mm512_store_si512(buf + 16, _mm512_unpacklo_epi64(LB, HB));
    }
    const __m512i p = _mm512_set1_epi64((long long)F::P);
    A = _mm512_mask_sub_epi64(A, _mm512_cmpge_epu64_mask(A, p), A, p);
    B = _mm512_mask_sub_epi64(B, _mm512_cmpge_epu64_mask(B, p), B, p);
    _mm512_storeu_si512(st, _mm512_permutexvar_epi64(_mm512_setr_epi64(0, 2, 4, 6, 1, 3, 5, 7), A));
    _mm256_storeu_si256((__m256i*)(st + 8), _mm512_castsi512_si256(_mm512_permutexvar_epi64(_mm512_setr_epi64(0, 2, 4, 6, 0, 0, 0, 0), B)));
}

#undef MB_AVX512
#undef MB_AVX512_INLINE

}  // namespace mono512
}  // namespace mbhost
#endif
