// Monolith-64 permutation over Goldilocks: width 12, 4 bars, 6 rounds, 8-bit
// lookups (goldilocks-cuda-rs/src/cpu_monolith.rs:18-144, device twin
// cuda/monolith.cuh). Host and device.
//
//   permute = concrete_0 ; for r = 1..6: bars ; bricks ; concrete_r
//   bars     byte S-box on words 0..3 of the canonical state
//   bricks   s_i += s_{i-1}^2 for i = 11 down to 1
//   concrete circulant MDS (first row 7 23 8 26 13 10 9 7 6 22 21 8) + constants
//
// The concrete layer is formed on three limbs of 22, 22 and 20 bits: the weights' row sum is 160, so the sums of a limb
// stay below 2^30 and 32-bit arithmetic is exact. The circulant is split over Z[x] / (x^12 - 1) = (x^6 + 1)(x^3 + 1)(x^3 - 1):
//   out_i = P_i + M_i, out_{i+6} = P_i - M_i   (i < 6; P of s_j + s_{j+6}, M of s_j - s_{j+6})
//   P_i = A_i + B_i, P_{i+3} = A_i - B_i       (i < 3, the same once more)
// with the halves moved into the weights, which all become powers of two: M -1 8 1 2 -4 1 (negacyclic), A 16 16 8,
// B -8 -1 -1 (negacyclic). That is 84 additions and shift-additions a limb where the circulant on 32-bit halves took
// 288 multiply-adds with 64-bit results, which cost the multiply pipe two to three times as much each
// (2^18 compressions: 96 -> 61 us). Values are loose in [0, 2^64) between layers; words 0..3 are made canonical before the
// bars (the S-box acts on the canonical bit pattern), and the caller canonicalises what it stores.
#pragma once
#include "gl_fast.cuh"

namespace gl {

#define GLMONO_RC_INIT                                                                                                  \
    {{0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0},                                                                               \
     {13596126580325903823ULL, 5676126986831820406ULL, 11349149288412960427ULL, 3368797843020733411ULL,                 \
      16240671731749717664ULL, 9273190757374900239ULL, 14446552112110239438ULL, 4033077683985131644ULL,                 \
      4291229347329361293ULL, 13231607645683636062ULL, 1383651072186713277ULL, 8898815177417587567ULL},                 \
     {2383619671172821638ULL, 6065528368924797662ULL, 16737578966352303081ULL, 2661700069680749654ULL,                  \
      7414030722730336790ULL, 18124970299993404776ULL, 9169923000283400738ULL, 15832813151034110977ULL,                 \
      16245117847613094506ULL, 11056181639108379773ULL, 10546400734398052938ULL, 8443860941261719174ULL},               \
     {15799082741422909885ULL, 13421235861052008152ULL, 15448208253823605561ULL, 2540286744040770964ULL,                \
      2895626806801935918ULL, 8644593510196221619ULL, 17722491003064835823ULL, 5166255496419771636ULL,                  \
      1015740739405252346ULL, 4400043467547597488ULL, 5176473243271652644ULL, 4517904634837939508ULL},                  \
     {18341030605319882173ULL, 13366339881666916534ULL, 6291492342503367536ULL, 10004214885638819819ULL,                \
      4748655089269860551ULL, 1520762444865670308ULL, 8393589389936386108ULL, 11025183333304586284ULL,                  \
      5993305003203422738ULL, 458912836931247573ULL, 5947003897778655410ULL, 17184667486285295106ULL},                  \
     {15710528677110011358ULL, 8929476121507374707ULL, 2351989866172789037ULL, 11264145846854799752ULL,                 \
      14924075362538455764ULL, 10107004551857451916ULL, 18325221206052792232ULL, 16751515052585522105ULL,               \
      15305034267720085905ULL, 15639149412312342017ULL, 14624541102106656564ULL, 3542311898554959098ULL},               \
     {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}}

constexpr int MONO_W = 12;
constexpr int MONO_ROUNDS = 6;

#ifdef __CUDACC__
static __constant__ uint64_t c_mono_rc[MONO_ROUNDS + 1][MONO_W] = GLMONO_RC_INIT;
#endif
static const uint64_t h_mono_rc[MONO_ROUNDS + 1][MONO_W] = GLMONO_RC_INIT;

GLF uint64_t mono_rc(int round, int i) {
#ifdef __CUDA_ARCH__
    return c_mono_rc[round][i];
#else
    return h_mono_rc[round][i];
#endif
}

// The byte S-box on four bytes at once: y = rotl8(x ^ (rotl8(~x,1) & rotl8(x,2) & rotl8(x,3)), 1). A rotation is two shifts and one choice by
// a mask.
GLF uint32_t mono_pick(uint32_t a, uint32_t b, uint32_t mask) { return (a & mask) | (b & ~mask); }
GLF uint32_t mono_bar32(uint32_t x) {
    const uint32_t l1 = mono_pick(x << 1, x >> 7, 0xFEFEFEFEu), l2 = mono_pick(x << 2, x >> 6, 0xFCFCFCFCu), l3 = mono_pick(x << 3, x >> 5, 0xF8F8F8F8u);
    const uint32_t t = x ^ (~l1 & l2 & l3);
    return mono_pick(t << 1, t >> 7, 0xFEFEFEFEu);
}
GLF uint64_t mono_bar(uint64_t x) { return pack64(mono_bar32(lo32(x)), mono_bar32(hi32(x))); }

// o = circulant times x, modulo 2^32.
GLF void mono_circulant(const uint32_t (&x)[MONO_W], uint32_t (&o)[MONO_W]) {
    uint32_t p[6], m[6], u[3], v[3], A[3], B[3], M[6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        p[j] = x[j] + x[j + 6];
        m[j] = x[j] - x[j + 6];
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        u[j] = p[j] + p[j + 3];
        v[j] = p[j] - p[j + 3];
    }
    const uint32_t sum16 = (u[0] + u[1] + u[2]) << 4;
#pragma unroll
    for (int i = 0; i < 3; i++) A[i] = sum16 - (u[(i + 2) % 3] << 3);
    B[0] = 0u - v[1] - v[2] - (v[0] << 3);
    B[1] = v[0] - v[2] - (v[1] << 3);
    B[2] = v[0] + v[1] - (v[2] << 3);
    M[0] = m[2] + m[5] - m[0] + (m[1] << 3) + (m[3] << 1) - (m[4] << 2);
    M[1] = m[3] - m[0] - m[1] + (m[2] << 3) + (m[4] << 1) - (m[5] << 2);
    M[2] = m[4] - m[1] - m[2] + (m[3] << 3) + (m[5] << 1) + (m[0] << 2);
    M[3] = m[5] - m[2] - m[3] + (m[4] << 3) - (m[0] << 1) + (m[1] << 2);
    M[4] = 0u - m[0] - m[3] - m[4] + (m[5] << 3) - (m[1] << 1) + (m[2] << 2);
    M[5] = 0u - m[1] - m[4] - m[5] - (m[0] << 3) - (m[2] << 1) + (m[3] << 2);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const uint32_t lo = A[i] + B[i], hi = A[i] - B[i];
        o[i] = lo + M[i];
        o[i + 6] = lo - M[i];
        o[i + 3] = hi + M[i + 3];
        o[i + 9] = hi - M[i + 3];
    }
}

// MDS times state plus the constants of `round` (`HAS_RC` false: zero constants).
template <bool HAS_RC>
GLF void mono_concrete(uint64_t* s, int round) {
    constexpr uint32_t MASK = (1u << 22) - 1;
    uint32_t x[MONO_W], o[MONO_W], top[MONO_W];
    uint64_t low[MONO_W];
#pragma unroll
    for (int j = 0; j < MONO_W; j++) x[j] = lo32(s[j]) & MASK;
    mono_circulant(x, o);
#pragma unroll
    for (int j = 0; j < MONO_W; j++) {
        low[j] = o[j];
        x[j] = (uint32_t)(s[j] >> 22) & MASK;
        top[j] = hi32(s[j]) >> 12;
    }
    mono_circulant(x, o);
#pragma unroll
    for (int j = 0; j < MONO_W; j++) low[j] = madwide(o[j], 1u << 22, low[j]);
    mono_circulant(top, o);
#pragma unroll
    for (int j = 0; j < MONO_W; j++) {
        uint64_t H = (uint64_t)o[j] << 12;
        if (HAS_RC) {   // the constant's halves: both sums stay below 2^54
            const uint64_t rc = mono_rc(round, j);
            low[j] += lo32(rc);
            H += hi32(rc);
        }
        s[j] = reduce_limb_sums(low[j], H);
    }
}

// In place; loose in, loose out.
GLF void monolith_permute(uint64_t* s) {
    mono_concrete<false>(s, 0);
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int r = 1; r <= MONO_ROUNDS; r++) {
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = mono_bar(canon(s[i]));
#pragma unroll
        for (int i = MONO_W - 1; i >= 1; i--) s[i] = mul_add(s[i - 1], s[i - 1], s[i]);
        if (r < MONO_ROUNDS) mono_concrete<true>(s, r);
        else mono_concrete<false>(s, r);
    }
}

#ifdef __CUDACC__
// ---- one permutation per thread, throughput form ---------------------------------------
// The linear layers on the FP64 pipe (halves of 32 bits: sums below 2^40), 192 of its operations a layer where the integer pipes took three
// limbs of 84 additions, their masks and their sums. As in Poseidon2's throughput form the rare repairs are left out and told of; the
// caller runs the exact form then. 7.4 k -> 6.2 k cycles a warp of permutations and scheduler (2^21 nodes: 428 -> 360 us), issue slots
// 0.68, the carry pipe 0.6 and the FP64 pipe 0.42 busy.
namespace monot {
using namespace fast;
struct RoundConstants {
    double half[MONO_ROUNDS + 1][MONO_W][2];
};
constexpr RoundConstants round_constants() {
    constexpr uint64_t rc[MONO_ROUNDS + 1][MONO_W] = GLMONO_RC_INIT;
    RoundConstants c{};
    for (int r = 0; r <= MONO_ROUNDS; r++)
        for (int i = 0; i < MONO_W; i++) {
            c.half[r][i][0] = LOW_HALF + (double)(rc[r][i] & 0xFFFFFFFFu);
            c.half[r][i][1] = HIGH_HALF + (double)(rc[r][i] >> 32);
        }
    return c;
}
static __constant__ RoundConstants d_round_constants = round_constants();

// o = circulant times the words x: mono_circulant's split, the differences x_j - x_(j+6) straight from 2^52 + x.
__device__ __forceinline__ void circulant(const uint32_t (&x)[MONO_W], double (&o)[MONO_W]) {
    double p[6], m[6], u[3], v[3], A[3], B[3], M[6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const double a = whole(x[j]), b = whole(x[j + 6]);
        m[j] = __dsub_rn(a, b);
        p[j] = __dadd_rn(__dadd_rn(a, -2 * TWO_52), b);
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        u[j] = __dadd_rn(p[j], p[j + 3]);
        v[j] = __dsub_rn(p[j], p[j + 3]);
    }
    const double sum16 = __dmul_rn(__dadd_rn(__dadd_rn(u[0], u[1]), u[2]), 16.0);
#pragma unroll
    for (int i = 0; i < 3; i++) A[i] = __fma_rn(u[(i + 2) % 3], -8.0, sum16);
    B[0] = __dsub_rn(__fma_rn(v[0], -8.0, -v[1]), v[2]);
    B[1] = __dsub_rn(__fma_rn(v[1], -8.0, v[0]), v[2]);
    B[2] = __dadd_rn(__fma_rn(v[2], -8.0, v[0]), v[1]);
    const auto row = [](double a, double b, double c, double by8, double by2, double by4, double two, double four) {
        return __fma_rn(by4, four, __fma_rn(by2, two, __fma_rn(by8, 8.0, __dadd_rn(__dadd_rn(a, b), c))));
    };
    M[0] = row(m[2], m[5], -m[0], m[1], m[3], m[4], 2.0, -4.0);
    M[1] = row(m[3], -m[0], -m[1], m[2], m[4], m[5], 2.0, -4.0);
    M[2] = row(m[4], -m[1], -m[2], m[3], m[5], m[0], 2.0, 4.0);
    M[3] = row(m[5], -m[2], -m[3], m[4], m[0], m[1], -2.0, 4.0);
    M[4] = row(-m[0], -m[3], -m[4], m[5], m[1], m[2], -2.0, 4.0);
    M[5] = row(-m[1], -m[4], -m[5], -m[0], m[2], m[3], -2.0, 4.0);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double lo = __dadd_rn(A[i], B[i]), hi = __dsub_rn(A[i], B[i]);
        o[i] = __dadd_rn(lo, M[i]);
        o[i + 6] = __dsub_rn(lo, M[i]);
        o[i + 3] = __dadd_rn(hi, M[i + 3]);
        o[i + 9] = __dsub_rn(hi, M[i + 3]);
    }
}
__device__ __forceinline__ void concrete(uint64_t* s, int round, Missed& missed) {
    uint32_t x[MONO_W];
    double l[MONO_W], h[MONO_W];
#pragma unroll
    for (int j = 0; j < MONO_W; j++) x[j] = lo32(s[j]);
    circulant(x, l);
#pragma unroll
    for (int j = 0; j < MONO_W; j++) x[j] = hi32(s[j]);
    circulant(x, h);
#pragma unroll
    for (int j = 0; j < MONO_W; j++)
        s[j] = from_halves(__dadd_rn(l[j], d_round_constants.half[round][j][0]), __dadd_rn(h[j], d_round_constants.half[round][j][1]), missed);
}
}  // namespace monot

// In place; loose in, loose out. False: the state is not the permutation's (run the exact form on the input again).
__device__ __forceinline__ bool monolith_permute_throughput(uint64_t* s) {
    fast::Missed missed{0, 0};
    monot::concrete(s, 0, missed);
#pragma unroll 1
    for (int r = 1; r <= MONO_ROUNDS; r++) {
#pragma unroll
        for (int i = 0; i < 4; i++) s[i] = mono_bar(canon(s[i]));
#pragma unroll
        for (int i = MONO_W - 1; i >= 1; i--) s[i] = fast::mul_add(s[i - 1], s[i - 1], s[i], missed);
        monot::concrete(s, r, missed);
    }
    return !missed.any();
}

// ---- one permutation spread over 16 lanes, or over a warp --------------------------------------
// For layers too small to fill the machine, where the latency of a permutation is what counts: lane i < 12 holds word i.
// A linear layer is twelve shuffles of each half against the lane's row of the circulant (instead of 288 multiply-adds), the bars
// run in lanes 0..3, the bricks take the neighbour's word by a shuffle. With a whole warp, the first sixteen lanes form the sums of the
// low halves and the other sixteen those of the high ones, and each hands the other its sum: half the shuffles and products. Rare
// repairs are left out; a warp that missed one runs the exact form, a permutation a thread. All 32 lanes of the warp must call.
// All layers above 2^8 digests 29.5 -> 23.6 us with the warp form where a block has a node a warp, 21 us with chained launches.
static __device__ const uint64_t g_mono_rc[MONO_ROUNDS + 1][MONO_W] = GLMONO_RC_INIT;   // per-lane reads
// C[(j - i) mod 12] = g_mono_row[12 - i + j]
static __device__ const uint32_t g_mono_row[2 * MONO_W] = {7, 23, 8, 26, 13, 10, 9, 7, 6, 22, 21, 8, 7, 23, 8, 26, 13, 10, 9, 7, 6, 22, 21, 8};
template <bool WARP>
__device__ __forceinline__ uint64_t mono_concrete_coop(uint64_t x, int lane, const uint32_t (&m)[MONO_W], uint64_t rc, fast::Missed& missed) {
    const uint32_t xl = lo32(x), xh = hi32(x);
    uint64_t L, H;
    if constexpr (WARP) {
        const bool high = lane >= 16;
        const uint32_t half = high ? xh : xl;
        uint64_t s[2] = {high ? hi32(rc) : lo32(rc), 0};
#pragma unroll
        for (int j = 0; j < MONO_W; j++) s[j & 1] = madwide(__shfl_sync(0xffffffffu, half, j, 16), m[j], s[j & 1]);
        const uint64_t mine = s[0] + s[1];
        const uint64_t other = pack64(__shfl_xor_sync(0xffffffffu, lo32(mine), 16), __shfl_xor_sync(0xffffffffu, hi32(mine), 16));
        L = high ? other : mine;
        H = high ? mine : other;
    } else {
        uint64_t l[2] = {lo32(rc), 0}, h[2] = {hi32(rc), 0};
#pragma unroll
        for (int j = 0; j < MONO_W; j++) {
            l[j & 1] = madwide(__shfl_sync(0xffffffffu, xl, j, 16), m[j], l[j & 1]);
            h[j & 1] = madwide(__shfl_sync(0xffffffffu, xh, j, 16), m[j], h[j & 1]);
        }
        L = l[0] + l[1];
        H = h[0] + h[1];
    }
    fast::Sum s;
    s.a = lo32(L);
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;" : "=&r"(s.b), "=r"(s.c) : "r"(hi32(L)), "r"(lo32(H)), "r"(hi32(H)));
    return fast::reduce(s, missed);
}
static __device__ __noinline__ uint64_t monolith_permute_gathered(uint64_t x, int lane16) {
    uint64_t s[MONO_W];
#pragma unroll
    for (int j = 0; j < MONO_W; j++) s[j] = pack64(__shfl_sync(0xffffffffu, lo32(x), j, 16), __shfl_sync(0xffffffffu, hi32(x), j, 16));
    monolith_permute(s);
#pragma unroll
    for (int j = 0; j < MONO_W; j++) x = j == lane16 ? s[j] : x;
    return x;
}
// x: word lane mod 16 (WARP: in two copies), zero from word 12 on
template <bool WARP>
__device__ __forceinline__ uint64_t monolith_permute_lanes(uint64_t x, int lane) {
    const uint64_t in = x;
    const int lane16 = lane & 15;
    const bool live = lane16 < MONO_W;
    fast::Missed missed{0, 0};
    uint32_t m[MONO_W];   // the lane's row of the circulant
#pragma unroll
    for (int j = 0; j < MONO_W; j++) m[j] = live ? g_mono_row[MONO_W - lane16 + j] : 0;
    x = mono_concrete_coop<WARP>(x, lane, m, 0, missed);
#pragma unroll 1
    for (int r = 1; r <= MONO_ROUNDS; r++) {
        const uint64_t b = mono_bar(canon(x));
        x = lane16 < 4 ? b : x;
        const uint64_t prev = pack64(__shfl_up_sync(0xffffffffu, lo32(x), 1, 16), __shfl_up_sync(0xffffffffu, hi32(x), 1, 16));
        const uint64_t y = fast::mul_add(prev, prev, x, missed);
        x = lane16 > 0 ? y : x;
        x = mono_concrete_coop<WARP>(x, lane, m, (live && r < MONO_ROUNDS) ? g_mono_rc[r][lane16] : 0, missed);
    }
    if (__any_sync(0xffffffffu, missed.any())) return monolith_permute_gathered(in, lane16);
    return x;
}
#endif

}  // namespace gl
