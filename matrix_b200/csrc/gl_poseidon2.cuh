// Poseidon2 permutation, width 8 over Goldilocks (4 + 22 + 4 rounds, x^7),
// plus the leaf / node hash forms used by the Merkle trees.
//
// Same function as the reference's poseidon2_permute_8 (cuda/poseidon2.cuh:322-358,
// CPU twin goldilocks-cuda-rs/src/cpu_poseidon2.rs:120-141) with the same round
// constants (cuda/poseidon2.cuh:50-94). State words are loose residues in
// [0, 2^64); callers canonicalise what they write out.
#pragma once
#include "gl_fast.cuh"

namespace gl {

#define GLP2_RC_EXT_INIT                                                                              \
    {                                                                                                 \
        {0xdd5743e7f2a5a5d9ULL, 0xcb3a864e58ada44bULL, 0xd5a3726889dedc0dULL, 0x79365a7f967583c1ULL,  \
         0xb7820c177b0a3c30ULL, 0x68a60479943b7240ULL, 0x0a22eeab67b97c41ULL, 0xbee9d90e037fa7d4ULL}, \
        {0xf1dda5b9259dfcb4ULL, 0x27515210be112d59ULL, 0x654a4db8f15f6c3aULL, 0x5a9bfff8c29db0c4ULL,  \
         0xb72f2628c95a885bULL, 0xffcb54fc166beaddULL, 0xe32f91d59c463772ULL, 0x9e0ff2a9bbea79dbULL}, \
        {0xce57d6245ddca6b2ULL, 0xb1fc8d402bba1eb1ULL, 0x64df974fb666d528ULL, 0x59e4e5b237e52e78ULL,  \
         0x5e255e2742caa8fcULL, 0xc4a17304e330ef9aULL, 0x60e3a513cdd9f0b1ULL, 0xbf29a6a5a0c9c8baULL}, \
        {0xcea721cce82fb11bULL, 0xe5b55eb8098ece81ULL, 0x4ec66bfb89f7c380ULL, 0xc33be12b6ef7e4faULL,  \
         0xa41b5f5b84c57d7dULL, 0xb526206b2138a936ULL, 0x9f7a5ac62f16eb4eULL, 0x7de77f405f683aa5ULL}, \
        {0x014ef1197d341346ULL, 0x9725e20825d07394ULL, 0xc8ff2a22516f3604ULL, 0xde1b51f7cf493493ULL,  \
         0xa7e3af1a53eadb78ULL, 0x9b7b7ee0ddf9f229ULL, 0xf0a460f2dc649e7dULL, 0xdc4448d02c2cb823ULL}, \
        {0xaa62c88e0b294011ULL, 0x058eb9d810ce9f74ULL, 0x4e3d7a5403566d24ULL, 0xe8ae66da2f8b7a63ULL,  \
         0x3fdad3b08dae2e0bULL, 0xec81e61303dd409bULL, 0x3cbaa1cd35d31fc4ULL, 0x847f7806eec88ffaULL}, \
        {0x98ae09a325893803ULL, 0xf8a6475077968838ULL, 0xdf55b7419443de5bULL, 0xdbe15699e696ca70ULL,  \
         0x8e54a27d8db00424ULL, 0x7679a45cd9d1e12aULL, 0x2844f52be73e0e2fULL, 0xd41f8eb31ada34f8ULL}, \
        {0xe9dd318bae1f3961ULL, 0xf7462137299efe1aULL, 0x6dbbe06779e1d573ULL, 0xfe35b05cbe707632ULL,  \
         0x5d8896b12654fd8cULL, 0x6f96ef47c32d4ae2ULL, 0xb0caa221dbbfc0daULL, 0x0bc2a5bf1f238d3fULL}, \
    }
#define GLP2_RC_INT_INIT                                                                             \
    {                                                                                                \
        0x488897d85ff51f56ULL, 0x1140737ccb162218ULL, 0xa7eeb9215866ed35ULL, 0x9bd2976fee49fcc9ULL,  \
        0xc0c8f0de580a3fccULL, 0x4fb2dae6ee8fc793ULL, 0x343a89f35f37395bULL, 0x223b525a77ca72c8ULL,  \
        0x56ccb62574aaa918ULL, 0xc4d507d8027af9edULL, 0xa080673cf0b7e95cULL, 0xf0184884eb70dcf8ULL,  \
        0x044f10b0cb3d5c69ULL, 0xe9e3f7993938f186ULL, 0x1b761c80e772f459ULL, 0x606cec607a1b5facULL,  \
        0x14a0c2e1d45f03cdULL, 0x4eace8855398574fULL, 0xf905ca7103eff3e6ULL, 0xf8c8f8d20862c059ULL,  \
        0xb524fe8bdd678e5aULL, 0xfbb7865901a1ec41ULL,                                                \
    }
#define GLP2_DIAG_INIT                                                                               \
    {                                                                                                \
        0xa98811a1fed4e3a5ULL, 0x1cc48b54f377e2a0ULL, 0xe40cd4f6c5609a26ULL, 0x11de79ebca97a4a3ULL,  \
        0x9177c73d8b7e929cULL, 0x2a6fe8085797e791ULL, 0x3de6e93329f8d5adULL, 0x3f7af9125da962feULL,  \
    }

// All table entries are below p. Statically initialised __constant__ data is
// loaded with the module on every device that runs it; no init call is needed.
static const uint64_t h_p2_rc_ext[8][8] = GLP2_RC_EXT_INIT;
static const uint64_t h_p2_rc_int[22] = GLP2_RC_INT_INIT;
static const uint64_t h_p2_diag[8] = GLP2_DIAG_INIT;
#ifdef __CUDACC__
static __constant__ uint64_t d_p2_rc_ext[8][8] = GLP2_RC_EXT_INIT;
static __constant__ uint64_t d_p2_rc_int[22] = GLP2_RC_INT_INIT;
static __constant__ uint64_t d_p2_diag[8] = GLP2_DIAG_INIT;
#endif

GLF uint64_t p2_rc_ext(int r, int i) {
#ifdef __CUDA_ARCH__
    return d_p2_rc_ext[r][i];
#else
    return h_p2_rc_ext[r][i];
#endif
}
GLF uint64_t p2_rc_int(int r) {
#ifdef __CUDA_ARCH__
    return d_p2_rc_int[r];
#else
    return h_p2_rc_int[r];
#endif
}
GLF uint64_t p2_diag(int i) {
#ifdef __CUDA_ARCH__
    return d_p2_diag[i];
#else
    return h_p2_diag[i];
#endif
}

GLF uint64_t sbox7(uint64_t x) {
    uint64_t x2 = sqr(x), x4 = sqr(x2), x3 = mul(x2, x);
    return mul(x4, x3);
}

// External linear layer: y = M x with M = [[2 M4, M4], [M4, 2 M4]],
// M4 = [2 3 1 1; 1 2 3 1; 1 1 2 3; 3 1 1 2] (the 4x4 map on each half followed
// by the cross-half sums of mds_light_8 in the reference), plus the next
// round's constants. Instead of a chain of modular additions, the low and high
// 32-bit halves of the eight inputs are accumulated separately with their small
// integer weights (row sum 21, so both sums stay below 2^37) and each output is
// reduced once.
template <bool HAS_RC>
GLF void p2_external_linear(uint64_t* s, int next_round) {
    constexpr uint32_t M[8][8] = {{4, 6, 2, 2, 2, 3, 1, 1}, {2, 4, 6, 2, 1, 2, 3, 1}, {2, 2, 4, 6, 1, 1, 2, 3},
                                  {6, 2, 2, 4, 3, 1, 1, 2}, {2, 3, 1, 1, 4, 6, 2, 2}, {1, 2, 3, 1, 2, 4, 6, 2},
                                  {1, 1, 2, 3, 2, 2, 4, 6}, {3, 1, 1, 2, 6, 2, 2, 4}};
    uint64_t y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint64_t L = 0, H = 0;
        if (HAS_RC) {
            uint64_t rc = p2_rc_ext(next_round, i);
            L = lo32(rc);
            H = hi32(rc);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            L = madwide(lo32(s[j]), M[i][j], L);
            H = madwide(hi32(s[j]), M[i][j], H);
        }
        y[i] = reduce_limb_sums(L, H);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = y[i];
}

// Internal linear layer: s_i = d_i s_i + sum(s); `rc0` (the next round's
// constant for lane 0, or 0) rides along in lane 0's sum.
GLF void p2_internal_linear(uint64_t* s, uint64_t rc0) {
    uint64_t SL = 0, SH = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        SL = madwide(lo32(s[i]), 1u, SL);
        SH = madwide(hi32(s[i]), 1u, SH);
    }
    uint64_t sum = reduce_limb_sums(SL, SH);
    s[0] = mul_add(s[0], p2_diag(0), add_c(sum, rc0));
#pragma unroll
    for (int i = 1; i < 8; i++) s[i] = mul_add(s[i], p2_diag(i), sum);
}

// In place; loose in, loose out. Round constants are added by the linear layer
// that precedes the S-boxes using them, so only the first external and the
// first internal / terminal constants need explicit additions. The exact form: what the throughput form below falls
// back to.
GLF void poseidon2_permute(uint64_t* s) {
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = add_c(s[i], p2_rc_ext(0, i));
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = sbox7(s[i]);
        if (r < 3) {
            p2_external_linear<true>(s, r + 1);
        } else {
            p2_external_linear<false>(s, 0);
            s[0] = add_c(s[0], p2_rc_int(0));
        }
    }
#pragma unroll 1
    for (int r = 0; r < 22; r++) {
        s[0] = sbox7(s[0]);
        p2_internal_linear(s, r < 21 ? p2_rc_int(r + 1) : 0);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = add_c(s[i], p2_rc_ext(4, i));
#pragma unroll 1
    for (int r = 4; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = sbox7(s[i]);
        if (r < 7) p2_external_linear<true>(s, r + 1);
        else p2_external_linear<false>(s, 0);
    }
}

#ifdef __CUDACC__
// ---- one permutation per thread, throughput form ---------------------------------------
// Bound by the integer pipes: 1436 to 2080 wide products (four cycles of the one pipe) and about as many carry additions (two of the
// other), which overlap to about 1.4. Against the exact form:
//   * the last repair of a reduction is left out. It is needed when a 64-bit word comes out below a 33-bit subtrahend (or
//     a sum of eight words has a high word within 64 of 2^32): about once in 2^31 products. Missed tells, and the caller runs the
//     exact form on the same input (one permutation in four million, half of them by words that only look like it);
//   * the sums of the internal layer are sums of whole words in 96 bits, three carry additions each; the external layers are on
//     the FP64 pipe.
// Exact form 25.3 k cycles per warp of permutations, carries counted and external layers in 96 bits 17.5 k, now 16.2 k (2^19
// permutations: 253 -> 236 us; tiles, which leave out the internal layers' products, 192 us).
namespace p2t {
using namespace fast;
__device__ __forceinline__ uint64_t sbox7(uint64_t x, Missed& missed) {
    const uint64_t x2 = mul(x, x, missed), x4 = mul(x2, x2, missed), x3 = mul(x2, x, missed);
    return mul(x4, x3, missed);
}
__device__ __forceinline__ uint64_t sbox7_soon(uint64_t x, Missed& missed) {
    const uint64_t x2 = sqr(x, missed), x4 = sqr(x2, missed), x3 = mul(x2, x, missed);
    return mul(x4, x3, missed);
}
// sums of words
__device__ __forceinline__ Sum sum(uint64_t x, uint64_t y) {
    Sum r;
    asm("add.cc.u32 %0, %3, %5;\n\taddc.cc.u32 %1, %4, %6;\n\taddc.u32 %2, 0, 0;"
        : "=&r"(r.a), "=&r"(r.b), "=r"(r.c) : "r"(lo32(x)), "r"(hi32(x)), "r"(lo32(y)), "r"(hi32(y)));
    return r;
}
__device__ __forceinline__ Sum sum(Sum x, uint64_t y) {
    Sum r;
    asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, 0;"
        : "=&r"(r.a), "=&r"(r.b), "=r"(r.c) : "r"(x.a), "r"(x.b), "r"(x.c), "r"(lo32(y)), "r"(hi32(y)));
    return r;
}
// The external layer on the FP64 pipe, which the integer work leaves idle: the 32-bit halves of the words are whole numbers in
// doubles (2^52 + x is the word 0x43300000 in front of x), their weighted sums (row sum 21) stay below 2^37, so every
// operation is exact, and 2^52 + sum carries the sum in its mantissa again. What is left to the integer pipes are the two
// words of each sum: 84 operations of the FP64 pipe take the place of 160 carry additions. A round with its S-boxes:
// 1286 -> 1064 cycles a warp and scheduler (990 with the shorter reduction).
// The constants' halves in front of round r (8: none), with what from_halves wants on the sums.
struct RoundConstants {
    double half[9][8][2];
};
constexpr RoundConstants round_constants() {
    constexpr uint64_t rc[8][8] = GLP2_RC_EXT_INIT;
    RoundConstants c{};
    for (int r = 0; r < 9; r++)
        for (int i = 0; i < 8; i++) {
            c.half[r][i][0] = LOW_HALF + (double)(r < 8 ? rc[r][i] & 0xFFFFFFFFu : 0);
            c.half[r][i][1] = HIGH_HALF + (double)(r < 8 ? rc[r][i] >> 32 : 0);
        }
    return c;
}
static __constant__ RoundConstants d_round_constants = round_constants();
__device__ __forceinline__ void external_linear(uint64_t* s, int next_round, Missed& missed) {
    double y[2][8];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        double v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __dadd_rn(whole(h ? hi32(s[i]) : lo32(s[i])), -TWO_52);
#pragma unroll
        for (int q = 0; q < 8; q += 4) {   // M4 on each half
            const double t01 = __dadd_rn(v[q], v[q + 1]), t23 = __dadd_rn(v[q + 2], v[q + 3]), t = __dadd_rn(t01, t23);
            const double t1 = __dadd_rn(t, v[q + 1]), t3 = __dadd_rn(t, v[q + 3]);
            y[h][q] = __dadd_rn(t1, t01);
            y[h][q + 1] = __fma_rn(2.0, v[q + 2], t1);
            y[h][q + 2] = __dadd_rn(t3, t23);
            y[h][q + 3] = __fma_rn(2.0, v[q], t3);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double a = y[h][i], b = y[h][i + 4];
            y[h][i] = __dadd_rn(__fma_rn(2.0, a, b), d_round_constants.half[next_round][i][h]);
            y[h][i + 4] = __dadd_rn(__fma_rn(2.0, b, a), d_round_constants.half[next_round][i + 4][h]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        s[i] = from_halves(y[0][i], y[1][i], missed);
    }
}
}  // namespace p2t

// In place; loose in, loose out. False: the state is not the permutation's (run the exact form on the input again).
__device__ __forceinline__ bool poseidon2_permute_throughput(uint64_t* s) {
    p2t::Missed missed{0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = add_c(s[i], p2_rc_ext(0, i));
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = p2t::sbox7(s[i], missed);
        p2t::external_linear(s, r < 3 ? r + 1 : 8, missed);
    }
    s[0] = add_c(s[0], p2_rc_int(0));
#pragma unroll 1
    for (int r = 0; r < 22; r++) {
        s[0] = p2t::sbox7(s[0], missed);
        p2t::Sum t = p2t::sum(s[0], s[1]);
#pragma unroll
        for (int i = 2; i < 8; i++) t = p2t::sum(t, s[i]);
        const uint64_t all = p2t::reduce(t, missed);
        s[0] = p2t::mul_add(s[0], p2_diag(0), r < 21 ? add_c(all, p2_rc_int(r + 1)) : all, missed);
#pragma unroll
        for (int i = 1; i < 8; i++) s[i] = p2t::mul_add(s[i], p2_diag(i), all, missed);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = add_c(s[i], p2_rc_ext(4, i));
#pragma unroll 1
    for (int r = 4; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = p2t::sbox7(s[i], missed);
        p2t::external_linear(s, r + 1, missed);
    }
    return !missed.any();
}

// ---- one permutation spread over 8 lanes ----------------------------------------
// Layers near the top of a Merkle tree (and a transcript) have too few
// permutations to fill the machine; what matters there is the latency of one
// permutation: the length of the chain of dependent instructions, 56 cycles for a product with its reduction, 24 for a
// shuffle. Eight consecutive lanes of a warp hold one state word each: the
// S-boxes of an external round run in parallel, the linear layers exchange
// words with warp shuffles. Per-lane constants come
// from global copies of the tables (a divergent index into __constant__ memory
// would serialise). All 32 lanes of the warp must call; `lane8` = lane & 7.
static __device__ const uint64_t g_p2_rc_ext[8][8] = GLP2_RC_EXT_INIT;
static __device__ const uint64_t g_p2_diag[8] = GLP2_DIAG_INIT;

// y = M x + rc over limbs of 22 bits (sums of weight 21 stay in 32), which butterflies of a lane's half and a shuffle across form: 208 cycles,
// 292 with every word sent to every lane and multiplied there.
__device__ __forceinline__ uint64_t p2_coop_external(uint64_t x, int lane8, uint64_t rc, p2t::Missed& missed) {
    const uint32_t limb[3] = {lo32(x) & 0x3FFFFFu, (uint32_t)(x >> 22) & 0x3FFFFFu, hi32(x) >> 12};
    const int next = (lane8 & 4) | ((lane8 + 1) & 3);
    uint32_t o[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t l = limb[k], r = __shfl_sync(0xffffffffu, l, next, 8);
        uint32_t t = l + __shfl_xor_sync(0xffffffffu, l, 1, 8);
        t += __shfl_xor_sync(0xffffffffu, t, 2, 8);
        const uint32_t y = t + l + 2 * r;   // M4 is circulant: first row 2 3 1 1
        o[k] = 2 * y + __shfl_xor_sync(0xffffffffu, y, 4, 8);
    }
    const uint64_t L = madwide(o[1], 1u << 22, (uint64_t)o[0]) + lo32(rc), H = madwide(o[2], 1u << 12, (uint64_t)hi32(rc));
    p2t::Sum s;
    s.a = lo32(L);
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;" : "=&r"(s.b), "=r"(s.c) : "r"(hi32(L)), "r"(lo32(H)), "r"(hi32(H)));
    return p2t::reduce(s, missed);
}

// The exact form for the whole warp, a permutation a thread: what the form below falls back to.
static __device__ __noinline__ uint64_t poseidon2_permute_gathered(uint64_t x, int lane8) {
    uint64_t s[8];
#pragma unroll
    for (int j = 0; j < 8; j++) s[j] = pack64(__shfl_sync(0xffffffffu, lo32(x), j, 8), __shfl_sync(0xffffffffu, hi32(x), j, 8));
    poseidon2_permute(s);
#pragma unroll
    for (int j = 0; j < 8; j++) x = j == lane8 ? s[j] : x;
    return x;
}

__device__ __forceinline__ uint64_t poseidon2_permute_coop8(uint64_t x, int lane8) {
    const uint64_t in = x;
    p2t::Missed missed{0, 0};
    x = add_c(x, g_p2_rc_ext[0][lane8]);
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
        x = p2t::sbox7_soon(x, missed);
        x = p2_coop_external(x, lane8, r < 3 ? g_p2_rc_ext[r + 1][lane8] : 0, missed);
    }
    // Internal rounds: y = (word 0 + constant)^7, words <- diag words + (y + the sum Q of words 1 .. 7). Every lane has the S-box
    // input s and forms y itself, so that no shuffle is on the chain from one S-box to the next:
    //     s <- (diag_0 + 1) y + Q + constant      four products deep
    // and Q, which needs the words one round late only, is formed beside the S-box: a three-step butterfly over limbs of
    // 22 bits (sums of eight stay in 32).
    const bool lane0 = lane8 == 0;
    const uint64_t diag = g_p2_diag[lane8], first = p2_diag(0) + 1;
    uint64_t s = add_c(pack64(__shfl_sync(0xffffffffu, lo32(x), 0, 8), __shfl_sync(0xffffffffu, hi32(x), 0, 8)), p2_rc_int(0));
#pragma unroll 1
    for (int r = 0; r < 22; r++) {
        const uint64_t y = p2t::sbox7_soon(s, missed);
        const uint64_t v = lane0 ? 0 : x;
        uint32_t l0 = lo32(v) & 0x3FFFFFu, l1 = (uint32_t)(v >> 22) & 0x3FFFFFu, l2 = hi32(v) >> 12;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            l0 += __shfl_xor_sync(0xffffffffu, l0, off, 8);
            l1 += __shfl_xor_sync(0xffffffffu, l1, off, 8);
            l2 += __shfl_xor_sync(0xffffffffu, l2, off, 8);
        }
        const uint64_t q = reduce_limb_sums(madwide(l1, 1u << 22, l0), (uint64_t)l2 << 12);
        const unsigned __int128 beside = (unsigned __int128)x * diag + q;
        const uint64_t qc = r < 21 ? add_c(q, p2_rc_int(r + 1)) : q;
        s = p2t::mul_add(y, first, qc, missed);
        x = p2t::reduce(beside + y, missed);   // below 2^128: diag < p
    }
    x = add_c(lane0 ? s : x, g_p2_rc_ext[4][lane8]);
#pragma unroll 1
    for (int r = 4; r < 8; r++) {
        x = p2t::sbox7_soon(x, missed);
        x = p2_coop_external(x, lane8, r < 7 ? g_p2_rc_ext[r + 1][lane8] : 0, missed);
    }
    if (__any_sync(0xffffffffu, missed.any())) return poseidon2_permute_gathered(in, lane8);
    return x;
}
#endif

}  // namespace gl
