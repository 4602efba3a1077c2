// The internal rounds of Poseidon2 (width 8 over Goldilocks) as a chain of S-boxes and sums: coefficients, from the tables of the
// permutation, and the permutation by a whole warp.
//
// In the 22 internal rounds only lane 0 passes an S-box, so everything else is linear in the words z before them (the S-box
// outputs of the fourth external round) and in the S-box inputs x_1 .. x_22 (x_22: word 0 after the rounds). With units
// x_r = scale[r] u_r chosen so that no S-box output needs a factor,
//     u_(r+1) = u_r^7 + R_(r+1),   R_r = const + sum_m row[r][z_m] z_m + sum_(q < r) row[r][u_q] u_q,
// and the other seven words after the rounds are sums of the same kind (scale[22] = 1; 7 divides no p - 1, so scale[0] is found
// backwards by seventh roots).
#pragma once
#include "gl_poseidon2.cuh"

namespace mb {
namespace mk {

constexpr uint64_t p2_mulmod(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % gl::P); }
constexpr uint64_t p2_addmod(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a + b) % gl::P); }
constexpr uint64_t p2_power(uint64_t a, uint64_t e) {
    uint64_t r = 1;
    for (; e; e >>= 1, a = p2_mulmod(a, a))
        if (e & 1) r = p2_mulmod(r, a);
    return r;
}
// One symbol's coefficients: s, the state's words as multiples of it in front of round `round`'s S-box (or, in_lane0, of its
// linear layer) become those after the rounds; x[r]: its part of the S-box input of round r, which y_r replaces; x[22]: s[0].
constexpr void p2_follow(uint64_t (&s)[8], int round, bool in_lane0, uint64_t (&x)[23]) {
    constexpr uint64_t diag[8] = GLP2_DIAG_INIT;
    for (int r = round; r < 22; r++) {
        if (r > round || !in_lane0) {
            x[r] = s[0];
            s[0] = 0;
        }
        uint64_t all = 0;
        for (int i = 0; i < 8; i++) all = p2_addmod(all, s[i]);
        for (int i = 0; i < 8; i++) s[i] = p2_addmod(p2_mulmod(s[i], diag[i]), all);
    }
    x[22] = s[0];
}
// Rows 0 .. 22: R_r; rows 23 .. 29: words 1 .. 7 after the rounds. Columns: a constant, z_0 .. z_7, u_1 .. u_22.
struct P2Linear {
    uint64_t row[30][31];
};
constexpr P2Linear p2_linear() {
    constexpr uint64_t m4[4] = {2, 3, 1, 1}, rc_int[22] = GLP2_RC_INT_INIT, rc_ext[8][8] = GLP2_RC_EXT_INIT;
    P2Linear p{};
    for (int r = 0; r < 30; r++) p.row[r][0] = r < 22 ? rc_int[r] : rc_ext[4][r - 22];
    for (int m = 0; m < 8; m++) {   // z_m goes through the external layer first
        uint64_t s[8] = {}, x[23] = {};
        for (int i = 0; i < 8; i++) s[i] = m4[(m - i + 8) & 3] * ((m >> 2) == (i >> 2) ? 2 : 1);
        p2_follow(s, 0, false, x);
        for (int r = 0; r < 30; r++) p.row[r][1 + m] = r < 23 ? x[r] : s[r - 22];
    }
    uint64_t of_y[30][22] = {};   // what y_q adds
    for (int q = 0; q < 22; q++) {
        uint64_t s[8] = {1, 0, 0, 0, 0, 0, 0, 0}, x[23] = {};
        p2_follow(s, q, true, x);
        for (int r = q + 1; r < 23; r++) of_y[r][q] = x[r];
        for (int i = 1; i < 8; i++) of_y[22 + i][q] = s[i];
    }
    // scales, from the last: scale[r + 1] = beta scale[r]^7, where y_r adds beta to x_(r+1); 1/7 is an exponent mod p - 1
    const uint64_t over = p2_power(of_y[1][0], gl::P - 2);
    uint64_t seventh = 0, scale[23] = {};
    for (int k = 1; k < 7; k++)
        if (((unsigned __int128)k * (gl::P - 1) + 1) % 7 == 0) seventh = (uint64_t)(((unsigned __int128)k * (gl::P - 1) + 1) / 7);
    scale[22] = 1;
    for (int r = 21; r >= 0; r--) scale[r] = p2_power(p2_mulmod(scale[r + 1], over), seventh);
    // y_q = scale[q]^7 u_q^7 = scale[q + 1] over (u_(q+1) - R_(q+1))
    for (int r = 0; r < 30; r++) {
        for (int q = 0; q < (r < 22 ? r - 1 : r == 22 ? 21 : 22); q++) {
            const uint64_t c = p2_mulmod(of_y[r][q], p2_mulmod(scale[q + 1], over)), minus = gl::P - c;
            for (int j = 0; j < 9 + q; j++) p.row[r][j] = p2_addmod(p.row[r][j], p2_mulmod(minus, p.row[q + 1][j]));
            p.row[r][9 + q] = p2_addmod(p.row[r][9 + q], c);
        }
        if (r < 22) {
            const uint64_t unit = p2_power(scale[r], gl::P - 2);
            for (int j = 0; j < 31; j++) p.row[r][j] = p2_mulmod(p.row[r][j], unit);
        }
    }
    return p;
}
constexpr P2Linear P2_LINEAR = p2_linear();

// ---- one permutation a warp -----------------------------------------------------------------------------------
// For layers that leave schedulers without a warp. Lane n keeps the sum of row n (30 rows) and adds to it each u as it becomes known, one
// product; every lane makes the S-boxes itself. R_(r+1) without u_r's part is whole one round ahead, so its reduction and its
// shuffle run beside the S-box, and the chain from u_r to u_(r+1) is the S-box alone: 9.1 k cycles a permutation against 12.0 k
// with eight lanes (13.3 k with lane 0's S-box output sent round), at one warp a scheduler.
struct alignas(16) P2Warp {   // copied 16 bytes at a time
    uint64_t z[8][32], c[32], u[23][32], own[22];   // by lane; own[q]: u_q to R_(q+1), which u[q] leaves out
};
constexpr P2Warp p2_warp(const P2Linear& p) {
    P2Warp w{};
    for (int n = 0; n < 30; n++) {
        w.c[n] = p.row[n][0];
        for (int m = 0; m < 8; m++) w.z[m][n] = p.row[n][1 + m];
        for (int q = 1; q < 23; q++)
            if (n >= 23 || n >= q + 2) w.u[q][n] = p.row[n][8 + q];
    }
    for (int q = 1; q < 22; q++) w.own[q] = p.row[q + 1][8 + q];
    return w;
}
static_assert(sizeof(P2Warp) % 16 == 0, "whole copies");
static __device__ const P2Warp g_p2_warp = p2_warp(P2_LINEAR);

__device__ __forceinline__ uint64_t p2_from_lane(uint64_t x, int lane) {
    return gl::pack64(__shfl_sync(0xffffffffu, gl::lo32(x), lane), __shfl_sync(0xffffffffu, gl::hi32(x), lane));
}
__device__ __forceinline__ uint64_t p2_reduce(const gl::Acc& s, gl::p2t::Missed& missed) {
    return gl::p2t::reduce(s.a0, s.a1, s.a2, s.a3, s.a4, missed);
}
__device__ __forceinline__ void p2_add(gl::Acc& a, const gl::Acc& b) {
    asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\taddc.cc.u32 %3, %3, %8;\n\taddc.u32 %4, %4, %9;"
        : "+r"(a.a0), "+r"(a.a1), "+r"(a.a2), "+r"(a.a3), "+r"(a.a4) : "r"(b.a0), "r"(b.a1), "r"(b.a2), "r"(b.a3), "r"(b.a4));
}
__device__ __forceinline__ gl::Acc p2_product(uint64_t a, uint64_t b) {
    const unsigned __int128 f = (unsigned __int128)a * b;
    const uint64_t lo = (uint64_t)f, hi = (uint64_t)(f >> 64);
    return gl::Acc{gl::lo32(lo), gl::hi32(lo), gl::lo32(hi), gl::hi32(hi), 0};
}
// x: word lane mod 8, in four copies; the same on return. w: g_p2_warp, in shared memory once ready() has been called. All 32 lanes call.
template <class Ready>
__device__ __forceinline__ uint64_t poseidon2_permute_warp(uint64_t x, int lane, const P2Warp& w, Ready ready) {
    const uint64_t in = x;
    const int lane8 = lane & 7;
    gl::p2t::Missed missed{0, 0};
    x = gl::add_c(x, gl::g_p2_rc_ext[0][lane8]);
#pragma unroll 1
    for (int r = 0; r < 3; r++) x = gl::p2_coop_external(gl::p2t::sbox7_soon(x, missed), lane8, gl::g_p2_rc_ext[r + 1][lane8], missed);
    x = gl::p2t::sbox7_soon(x, missed);
    ready();
    gl::Acc sum = gl::acc_from(w.c[lane]), odd = gl::acc_zero();
#pragma unroll
    for (int m = 0; m < 8; m += 2) {
        gl::acc_mul(sum, w.z[m][lane], p2_from_lane(x, m));
        gl::acc_mul(odd, w.z[m + 1][lane], p2_from_lane(x, m + 1));
    }
    p2_add(sum, odd);
    uint64_t u = p2_reduce(sum, missed), ahead = p2_from_lane(u, 1);   // R_0 and R_1
    u = p2_from_lane(u, 0);
    uint64_t coefficient = w.u[0][lane], own = w.own[0];
#pragma unroll 1
    for (int q = 0; q < 22; q++) {
        const uint64_t u2 = gl::p2t::sqr(u, missed), u4 = gl::p2t::sqr(u2, missed), u3 = gl::p2t::mul(u2, u, missed);
        gl::Acc next = gl::acc_from(ahead);
        gl::acc_mul(next, own, u);
        gl::acc_mul(sum, coefficient, u);
        ahead = p2_from_lane(p2_reduce(sum, missed), q + 2);   // R_(q+2) up to u_q
        coefficient = w.u[q + 1][lane];
        own = w.own[q < 21 ? q + 1 : 21];
        p2_add(next, p2_product(u4, u3));
        u = p2_reduce(next, missed);
    }
    gl::acc_mul(sum, coefficient, u);
    x = p2_from_lane(p2_reduce(sum, missed), 22 + lane8);
    x = lane8 ? x : u;
#pragma unroll 1
    for (int r = 4; r < 8; r++) x = gl::p2_coop_external(gl::p2t::sbox7_soon(x, missed), lane8, r < 7 ? gl::g_p2_rc_ext[r + 1][lane8] : 0, missed);
    if (__any_sync(0xffffffffu, missed.any(29)))   // a row: at most thirty products
        return gl::poseidon2_permute_gathered(in, lane8);
    return x;
}

}  // namespace mk
}  // namespace mb
