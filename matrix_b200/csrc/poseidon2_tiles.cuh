// Poseidon2 over tiles of 128 permutations with the internal rounds' linear algebra on the tensor cores.
//
// In the 22 internal rounds only lane 0 passes an S-box, so everything else is linear in the words z before them (the S-box
// outputs of the fourth external round) and the S-box outputs y_0 .. y_21: the S-box inputs are
//     x_r = c_r + sum_m alpha[r][m] z_m + sum_(q < r) beta[r - q] y_q,
// the words after the rounds are sum_m omega[i][m] z_m + sum_q gamma[q][i] y_q. A permutation a thread, the rounds' 176 products
// by the diagonal and their sums are a third of its time. As contractions over bytes (a row of the operand: the bytes
// of one permutation's words, the other operand: the bytes of 2^(8 i) times a coefficient mod p) they cost the tensor pipe
// about 900 of the 14 k cycles that the 128 permutations take the SM, and a thread: eight 32-bit sums to put together and
// reduce per x_r and word (27 instructions, 30 of them), and 1.5 products a round, because four y at a time go into the
// operand (32 bytes, one step of K) and those of the same four are added by hand.
//
// A block of six tiles an SM; a tile's 240 columns of sums stay in tensor memory over its internal rounds, so two tiles are
// there at a time (in a fixed order: tile g has half g mod 2 after tile g - 2 or g + 4), while the others are in their external
// rounds. Every wait is bounded; once one ran out, the whole block takes the exact form.
// Layers of 2^23 permutations: 17.1 k -> 14.7 k cycles a warp of permutations (3978 -> 3432 us).
#pragma once
#include "gl_poseidon2.cuh"
#include "tcgen05.cuh"

namespace mb {
namespace mk {

// ---- the coefficients, from the tables of the permutation -------------------------------------------
struct P2Linear {
    uint64_t alpha[22][8], omega[8][8], beta[22], gamma[22][8];   // beta[0] is not used
};
constexpr uint64_t p2_mulmod(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % gl::P); }
constexpr uint64_t p2_addmod(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a + b) % gl::P); }
// One symbol's coefficients: s, the state's words as multiples of it in front of round `round`'s S-box (or, in_lane0, of its
// linear layer) become those after the rounds; x[r]: its part of the S-box input of round r, which y_r replaces.
constexpr void p2_follow(uint64_t (&s)[8], int round, bool in_lane0, uint64_t (&x)[22]) {
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
}
constexpr P2Linear p2_linear() {
    P2Linear p{};
    constexpr uint64_t m4[4] = {2, 3, 1, 1};
    for (int m = 0; m < 8; m++) {   // z_m goes through the external layer first
        uint64_t s[8] = {}, x[22] = {};
        for (int i = 0; i < 8; i++) s[i] = m4[(m - i + 8) & 3] * ((m >> 2) == (i >> 2) ? 2 : 1);
        p2_follow(s, 0, false, x);
        for (int r = 0; r < 22; r++) p.alpha[r][m] = x[r];
        for (int i = 0; i < 8; i++) p.omega[i][m] = s[i];
    }
    for (int q = 0; q < 22; q++) {
        uint64_t s[8] = {1, 0, 0, 0, 0, 0, 0, 0}, x[22] = {};
        p2_follow(s, q, true, x);
        for (int i = 0; i < 8; i++) p.gamma[q][i] = s[i];
        if (q == 0)
            for (int r = 1; r < 22; r++) p.beta[r] = x[r];
    }
    return p;
}
static __device__ const P2Linear g_p2_linear = p2_linear();
static __constant__ uint64_t d_p2_beta[4] = {0, p2_linear().beta[1], p2_linear().beta[2], p2_linear().beta[3]};

// ---- operands: 16-byte units by column, the rows of a column one after another --------------------------
constexpr int P2_TILES = 6, P2_TILE = 128, P2_BLK = P2_TILES * P2_TILE;
constexpr uint32_t P2_X = 22 * 8, P2_N = P2_X + 64;                 // columns: the bytes of x_r, then of the words after
constexpr uint32_t P2_Z = 0, P2_Y = P2_Z + P2_N * 64, P2_O = P2_Y + 144 * 32, P2_CONST = P2_O + 6 * 64 * 32;
constexpr uint32_t P2_SMEM = P2_CONST + P2_TILES * P2_TILE * 64;

__device__ __forceinline__ uint64_t p2_desc(uint32_t saddr, uint32_t rows) {   // K-major, no swizzle
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)rows << 16) | ((uint64_t)(128 >> 4) << 32) | (1ULL << 46);
}
// the eight bytes of 2^(8 i) c for every i: rows row .. row + 7, bytes k .. k + 7 of an operand with `rows` rows
__device__ __forceinline__ void p2_place(uint8_t* op, uint32_t rows, uint32_t row, uint32_t k, uint64_t c) {
#pragma unroll 1
    for (uint32_t i = 0; i < 8; i++) {
        const uint64_t f = gl::canon(gl::mul(c, 1ULL << (8 * i)));
        uint8_t* p = op + ((k + i) >> 4) * rows * 16 + ((k + i) & 15);
#pragma unroll
        for (uint32_t b = 0; b < 8; b++) p[16 * (row + b)] = (uint8_t)(f >> (8 * b));
    }
}
__device__ __forceinline__ void p2_operands(uint8_t* sm) {
    for (int x = threadIdx.x; x < 240 + 72 + 192; x += P2_BLK) {
        if (x < 240) {
            const int n = x >> 3, m = x & 7;
            p2_place(sm + P2_Z, P2_N, 8 * n, 8 * m, n < 22 ? g_p2_linear.alpha[n][m] : g_p2_linear.omega[n - 22][m]);
        } else if (x < 312) {   // x_(4 b + d) from y_(4 b - 4 + j), the same for every b
            const int d = (x - 240) >> 2, j = (x - 240) & 3;
            p2_place(sm + P2_Y, 144, 8 * d, 8 * j, g_p2_linear.beta[d + 4 - j]);
        } else {
            const int b = (x - 312) >> 5, i = (x >> 2) & 7, j = x & 3, q = 4 * b + j;   // 312 is a multiple of four
            p2_place(sm + P2_O + b * 64 * 32, 64, 8 * i, 8 * j, q < 22 ? g_p2_linear.gamma[q][i] : 0);
        }
    }
}

// ---- a tile's internal rounds -------------------------------------------------------------------------------
// sum_k s[k] 2^(8 k) + c, three limbs: s[k] <= 255^2 * 240
__device__ __forceinline__ gl::Acc p2_bytes(const uint32_t* s, uint64_t c) {
    const uint64_t u = gl::pack64(s[0], s[4]) + (gl::pack64(s[1], s[5]) << 8), w = gl::pack64(s[2], s[6]) + (gl::pack64(s[3], s[7]) << 8);
    gl::Acc a{gl::lo32(u), gl::hi32(u), 0, 0, 0};
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %5, 0;\n\t"
        "add.cc.u32 %0, %0, %6;\n\taddc.cc.u32 %1, %1, %7;\n\taddc.u32 %2, %2, 0;"
        : "+r"(a.a0), "+r"(a.a1), "+r"(a.a2)
        : "r"(gl::lo32(w << 16)), "r"(gl::hi32(w << 16)), "r"((uint32_t)(w >> 48)), "r"(gl::lo32(c)), "r"(gl::hi32(c)));
    return a;
}
// gl::acc_reduce without its repair (p2t::reduce)
__device__ __forceinline__ uint64_t p2_reduce(const gl::Acc& s, gl::p2t::Missed& missed) {
    uint32_t A, c, B0, B1, r0, r1;
    asm("add.cc.u32 %0, %4, %5;\n\taddc.u32 %1, 0, 0;\n\taddc.cc.u32 %2, %5, %6;\n\taddc.u32 %3, %7, 0;"
        : "=&r"(A), "=&r"(c), "=&r"(B0), "=r"(B1) : "r"(s.a1), "r"(s.a2), "r"(s.a3), "r"(s.a4));
    A += c;
    asm("sub.cc.u32 %0, %3, %4;\n\tsubc.cc.u32 %1, %5, %6;\n\tsubc.u32 %2, %2, 0;"
        : "=&r"(r0), "=r"(r1), "+r"(missed.borrows) : "r"(s.a0), "r"(B0), "r"(A), "r"(B1));
    return gl::pack64(r0, r1);
}

struct P2Tile {
    uint32_t tmem;        // its half of tensor memory, at the warp's lanes
    uint32_t consts;      // shared address of the operands of coefficients
    uint8_t* rows;        // its operand: unit c of row r at 2048 c + 16 r
    // mbarriers: its MMAs; it is through with its half of tensor memory; the tile before it there is
    uint32_t done, free, before;
    uint32_t row;         // the thread in the tile
    uint32_t id;          // named barrier
    int use;              // phase of `before` to wait for next, or negative
    uint32_t turn = 0;    // phases of `done`
    tc::Issued issued;    // row 0's MMAs, one commit a turn of `done`
    volatile int* failed; // the block's: a wait ran out
    __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) {
        if (!*failed && !tc::mbar_wait(bar, parity)) *failed = 1;
    }
    __device__ __forceinline__ void put(int unit, uint64_t a, uint64_t b) {
        *reinterpret_cast<ulonglong2*>(rows + 2048 * unit + 16 * row) = make_ulonglong2(a, b);
    }
    // the tile's rows are written and its sums read
    __device__ __forceinline__ void meet() {
        tc::fence_operands();
        tc::fence_before();
        tc::named_sync(P2_TILE, id);
        tc::fence_after();
    }
    __device__ __forceinline__ void finish() {
        wait(done, turn & 1);
        turn++;
        tc::fence_after();
    }
};

// s: the words after the fourth external round's S-boxes; on return the words before the fifth's, its constants added.
__device__ __forceinline__ void p2_internal_rounds(P2Tile& t, uint64_t* s, gl::p2t::Missed& missed) {
    const uint32_t ops = tc::smem_u32(t.rows), z = t.tmem & 0x0000FFFFu;
#pragma unroll
    for (int c = 0; c < 4; c++) t.put(c, s[2 * c], s[2 * c + 1]);
    if (t.use >= 0) t.wait(t.before, t.use & 1);
    t.meet();
    if (t.row == 0 && !*t.failed) {
#pragma unroll
        for (int ks = 0; ks < 2; ks++)
            tc::mma_i8(z, p2_desc(ops + 4096 * ks, 128), p2_desc(t.consts + P2_Z + ks * 32 * P2_N, P2_N), tc::idesc_u8(P2_N, false), ks > 0);
        t.issued.commit_to(t.done, t.turn);
    }
    t.finish();
#pragma unroll 1
    for (int b = 0; b < 6; b++) {
        uint64_t y[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[16];
            if (b == 5 && h == 1) break;
            tc::ld16(t.tmem + 32 * b + 16 * h, v);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = 2 * h + e;
                gl::Acc x = p2_bytes(v + 8 * e, gl::p2_rc_int(4 * b + j));
#pragma unroll
                for (int q = 0; q < j; q++) gl::acc_mul(x, d_p2_beta[j - q], y[q]);
                y[j] = gl::p2t::sbox7(p2_reduce(x, missed), missed);
            }
            t.put(h, y[2 * h], y[2 * h + 1]);
        }
        t.meet();
        if (t.row == 0 && !*t.failed) {
            const uint64_t rows = p2_desc(ops, 128);
            if (b < 5)
                tc::mma_i8(z + 32 * (b + 1), rows, p2_desc(t.consts + P2_Y, 144), tc::idesc_u8(0, false) | ((uint32_t)(18 - 4 * b) << 17), true);
            tc::mma_i8(z + P2_X, rows, p2_desc(t.consts + P2_O + b * 64 * 32, 64), tc::idesc_u8(64, false), true);
            t.issued.commit_to(t.done, t.turn);
        }
        t.finish();
    }
#pragma unroll
    for (int h = 0; h < 4; h++) {
        uint32_t v[16];
        tc::ld16(t.tmem + P2_X + 16 * h, v);
        s[2 * h] = p2_reduce(p2_bytes(v, gl::p2_rc_ext(4, 2 * h)), missed);
        s[2 * h + 1] = p2_reduce(p2_bytes(v + 8, gl::p2_rc_ext(4, 2 * h + 1)), missed);
    }
    tc::fence_before();
    __syncwarp();
    if ((t.row & 31) == 0) tc::mbar_arrive(t.free);
    t.use++;
}

// poseidon2_permute_throughput by a tile's threads together
__device__ __forceinline__ bool p2_permute_tile(P2Tile& t, uint64_t* s) {
    gl::p2t::Missed missed{0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = gl::add_c(s[i], gl::p2_rc_ext(0, i));
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = gl::p2t::sbox7(s[i], missed);
        gl::p2t::external_linear<true>(s, r + 1, missed);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = gl::p2t::sbox7(s[i], missed);
    p2_internal_rounds(t, s, missed);
#pragma unroll 1
    for (int r = 4; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = gl::p2t::sbox7(s[i], missed);
        if (r < 7) gl::p2t::external_linear<true>(s, r + 1, missed);
        else gl::p2t::external_linear<false>(s, 0, missed);
    }
    return (missed.borrows | missed.carries) == 0 && !*t.failed;
}

}  // namespace mk
}  // namespace mb
