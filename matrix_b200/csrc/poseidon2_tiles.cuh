// Poseidon2 over tiles of 128 permutations with the internal rounds' linear algebra on the tensor cores.
//
// With the sums of poseidon2_linear.cuh: as contractions over bytes (a row of the operand: the bytes of one permutation's words, the
// other operand: the bytes of 2^(8 i) times a coefficient mod p) the sums cost the tensor pipe about a tenth of the time that the 128
// permutations take the SM, and a thread: eight 32-bit sums to put together per R, in front of a reduction that the S-box's
// last product needs anyway. Four u at a time go into the operand (32 bytes, one step of K); of those of the same four,
// u_r to R_(r+1) makes the S-box u (u^6 + a), and the other three products are made by hand.
// The MMA that takes u_(4b) .. u_(4b+3) to the next R runs while a thread is in the S-box of u_(4b+3).
//
// A block of four tiles an SM, each with 128 columns of tensor memory: the sums of R_0 .. R_15 first, those of R_16 .. R_22
// and the other words, from all the operands so far, once these are read. Every wait is bounded; once one ran out, the whole
// block takes the exact form.
// Four tiles, because a tile is 128 threads of up to 128 registers and three leave schedulers idle (3237 us below).
// Bound by the integer pipes (ncu, 2^22 leaves: 0.67 of the multiply pipe, 0.51 of the logic pipe, 0.56 of the issue slots, 6940
// instructions a permutation). Layers of 2^23 permutations:
// 3426 us (14.9 k cycles a warp of permutations and scheduler) with six tiles of which two at a time had tensor memory, six products
// by hand in four rounds, every S-box output reduced apart and external layers of carry additions; 2917 us (12.7 k) now.
#pragma once
#include "poseidon2_linear.cuh"
#include "tcgen05.cuh"

namespace mb {
namespace mk {

// ---- the products by hand ---------------------------------------------------------------------------------
// By block of four, what its own u add: u_(4b), u_(4b+1), u_(4b+2) to the next one (own), u_(4b) to R_(4b+2), and
// u_(4b), u_(4b+1) to R_(4b+3).
struct P2Near {
    uint64_t own[6][3], far[6][3];
};
constexpr P2Near p2_near(const P2Linear& p) {
    P2Near n{};
    for (int b = 0; b < 6; b++) {
        for (int j = 0; j < 3; j++)
            if (4 * b + j > 0 && 4 * b + j < 22) n.own[b][j] = p.row[4 * b + 1 + j][8 + 4 * b + j];
        if (b > 0) n.far[b][0] = p.row[4 * b + 2][8 + 4 * b];
        if (b < 5) n.far[b][2] = p.row[4 * b + 3][9 + 4 * b];
        if (b > 0 && b < 5) n.far[b][1] = p.row[4 * b + 3][8 + 4 * b];
    }
    return n;
}
static __device__ const P2Linear g_p2_linear = P2_LINEAR;
static __constant__ P2Near d_p2_near = p2_near(P2_LINEAR);

// ---- operands: 16-byte units by column, the rows of a column one after another --------------------------
constexpr int P2_TILES = 4, P2_TILE = 128, P2_BLK = P2_TILES * P2_TILE;
// Columns of the two stages (eight a row): R_0 .. R_15; R_16 .. R_22 and the words 1 .. 7. Steps of K in the order of the table:
// z (two) to the first stage, to the second; chunk k = u_(4k) .. u_(4k+3) to the first stage's R_(4k+4) and later (k < 3), to the
// second stage (k < 4), chunk 4 from R_20 on, chunk 5 to the words (and zeros to R_22: N is a multiple of sixteen).
constexpr uint32_t P2_NA = 128, P2_NB = 112;
struct P2Step {
    uint32_t first, columns;   // row of P2Linear, columns
    uint32_t from;             // four symbols: z_(from), or u_(from - 8)
};
constexpr int P2_STEPS = 13;
__host__ __device__ constexpr P2Step p2_step(int i) {
    return i < 2 ? P2Step{0, P2_NA, 4u * i} : i < 4 ? P2Step{16, P2_NB, 4u * (i - 2)}
         : i < 7 ? P2Step{4u * (i - 3), P2_NA - 32u * (i - 3), 8 + 4u * (i - 4)}
         : i < 11 ? P2Step{16, P2_NB, 8 + 4u * (i - 7)} : i == 11 ? P2Step{20, 80, 24} : P2Step{22, 64, 28};
}
// where a step's operand lies, in rows of 32 bytes
__host__ __device__ constexpr uint32_t p2_at(int i) { return i == 0 ? 0 : p2_at(i - 1) + p2_step(i - 1).columns; }
constexpr uint32_t P2_TABLE_ROWS = p2_at(P2_STEPS);
struct alignas(16) P2Table {   // read 16 bytes at a time
    uint64_t word[4 * P2_TABLE_ROWS];
};
// Byte i of a symbol adds byte b of 2^(8 i) times its coefficient to column b: byte i of word [row of the column][symbol].
constexpr P2Table p2_table(const P2Linear& p) {
    P2Table t{};
    for (int st = 0; st < P2_STEPS; st++) {
        const P2Step step = p2_step(st);
        for (uint32_t n = 0; n < step.columns / 8; n++)
            for (uint32_t j = 0; j < 4; j++) {
                const uint32_t symbol = step.from + j, row = step.first + n, u = symbol - 8;
                // z as they are; u_0 is no symbol, and what a u adds to R of its own four is made by hand
                uint64_t c = symbol < 8 ? p.row[row][1 + symbol] : u >= 1 && u <= 22 && (row > 22 || row >= (u & ~3u) + 4) ? p.row[row][8 + u] : 0;
                uint64_t out[8] = {};
                for (int i = 0; i < 8; i++) {
                    for (int b = 0; b < 8; b++) out[b] |= (uint64_t)((c >> (8 * b)) & 0xFF) << (8 * i);
                    c = p2_mulmod(c, 256);
                }
                // 16-byte unit j / 2, its word j mod 2
                for (int b = 0; b < 8; b++) t.word[4 * p2_at(st) + ((j >> 1) * step.columns + 8 * n + b) * 2 + (j & 1)] = out[b];
            }
    }
    return t;
}
static_assert(sizeof(P2Table) % 16 == 0, "whole units");
static __device__ const P2Table g_p2_table = p2_table(P2_LINEAR);

// shared memory: the table, a column of ones and the constants for it (two stages), the tiles' operands (z, chunks 0 .. 3; 4 and 5 go
// where z was)
constexpr uint32_t P2_ONE = 32 * P2_TABLE_ROWS, P2_C = P2_ONE + 32 * P2_TILE, P2_ROWS = P2_C + 32 * (P2_NA + P2_NB), P2_UNITS = 12,
                   P2_SMEM = P2_ROWS + P2_BLK * 16 * P2_UNITS;

__device__ __forceinline__ uint64_t p2_desc(uint32_t saddr, uint32_t rows) {   // K-major, no swizzle
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)rows << 16) | ((uint64_t)(128 >> 4) << 32) | (1ULL << 46);
}
__device__ __forceinline__ void p2_operands(uint8_t* sm) {
    ulonglong2* p = reinterpret_cast<ulonglong2*>(sm);
    const ulonglong2* table = reinterpret_cast<const ulonglong2*>(g_p2_table.word);
    for (uint32_t x = threadIdx.x; x < 2 * P2_TABLE_ROWS; x += P2_BLK) p[x] = table[x];
    for (uint32_t x = threadIdx.x; x < 2 * P2_TILE; x += P2_BLK) p[P2_ONE / 16 + x] = make_ulonglong2(x < P2_TILE ? 1 : 0, 0);
    for (uint32_t x = threadIdx.x; x < P2_NA + P2_NB; x += P2_BLK) {   // a byte of a constant, times the one
        const uint32_t rows = x < P2_NA ? P2_NA : P2_NB, at = P2_C / 16 + (x < P2_NA ? x : P2_NA + x);
        p[at] = make_ulonglong2((g_p2_linear.row[x >> 3][0] >> (8 * (x & 7))) & 0xFF, 0);
        p[at + rows] = make_ulonglong2(0, 0);
    }
}

// ---- a tile's internal rounds -------------------------------------------------------------------------------
// a + sum_k s[k] 2^(8 k). s[k] <= 255^2 * 240 + 255, so that s[k] + 2^8 s[k + 1] is a word.
__device__ __forceinline__ void p2_add_bytes(gl::Acc& a, const uint32_t* s) {
    const uint32_t t0 = s[0] + (s[1] << 8), t1 = s[2] + (s[3] << 8), t2 = s[4] + (s[5] << 8), t3 = s[6] + (s[7] << 8);
    const uint64_t w = gl::pack64(t1, t3);
    uint32_t l0, l1, l2;
    asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;"
        : "=&r"(l0), "=&r"(l1), "=r"(l2) : "r"(t0), "r"(t1 << 16), "r"(t2), "r"((uint32_t)(w >> 16)), "r"(t3 >> 16));
    asm("add.cc.u32 %0, %0, %5;\n\taddc.cc.u32 %1, %1, %6;\n\taddc.cc.u32 %2, %2, %7;\n\taddc.cc.u32 %3, %3, 0;\n\taddc.u32 %4, %4, 0;"
        : "+r"(a.a0), "+r"(a.a1), "+r"(a.a2), "+r"(a.a3), "+r"(a.a4) : "r"(l0), "r"(l1), "r"(l2));
}
// u^7, and u^7 + a u, not reduced
__device__ __forceinline__ gl::Acc p2_seventh(uint64_t u, gl::p2t::Missed& missed) {
    const uint64_t u2 = gl::p2t::mul(u, u, missed);
    return p2_product(gl::p2t::mul(u2, u2, missed), gl::p2t::mul(u2, u, missed));
}
__device__ __forceinline__ gl::Acc p2_seventh_and(uint64_t u, uint64_t a, gl::p2t::Missed& missed) {
    const uint64_t u2 = gl::p2t::mul(u, u, missed), u3 = gl::p2t::mul(u2, u, missed);
    return p2_product(u, gl::p2t::mul_add(u3, u3, a, missed));
}
struct P2Tile {
    uint32_t tmem;        // its 128 columns of tensor memory, at the warp's lanes
    uint32_t consts;      // shared address of the table
    uint8_t* rows;        // its operand: unit c of row r at 2048 c + 16 r
    uint32_t done;        // mbarrier: its MMAs
    uint32_t row;         // the thread in the tile
    uint32_t id;          // named barrier
    uint32_t turn = 0;    // phases of `done`
    tc::Issued issued;    // row 0's MMAs, one commit a turn of `done`
    volatile int* failed; // the block's: a wait ran out
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
    // the columns from `column` on += units unit and unit + 1 of the rows, times a step of the table
    template <int STEP>
    __device__ __forceinline__ void add(int unit, uint32_t column) {
        constexpr uint32_t at = 32 * p2_at(STEP), columns = p2_step(STEP).columns;
        tc::mma_i8((tmem & 0x0000FFFFu) + column, p2_desc(tc::smem_u32(rows) + 2048 * unit, P2_TILE), p2_desc(consts + at, columns),
                   tc::idesc_u8(columns, false), true);
    }
    __device__ __forceinline__ void begin(bool second) {   // the constants
        const uint32_t columns = second ? P2_NB : P2_NA;
        tc::mma_i8(tmem & 0x0000FFFFu, p2_desc(consts + P2_ONE, P2_TILE), p2_desc(consts + P2_C + (second ? 32 * P2_NA : 0), columns),
                   tc::idesc_u8(columns, false), false);
    }
    __device__ __forceinline__ void finish() {
        if (!*failed && !tc::mbar_wait(done, turn & 1)) *failed = 1;
        turn++;
        tc::fence_after();
    }
};

// s: the words after the fourth external round's S-boxes; on return the words before the fifth's, its constants added.
__device__ __forceinline__ void p2_internal_rounds(P2Tile& t, uint64_t* s, gl::p2t::Missed& missed) {
#pragma unroll
    for (int c = 0; c < 4; c++) t.put(c, s[2 * c], s[2 * c + 1]);
    t.meet();
    if (t.row == 0 && !*t.failed) {
        t.begin(false);
        t.add<0>(0, 0);
        t.add<1>(2, 0);
        t.issued.commit_to(t.done, t.turn);
    }
    gl::Acc x = gl::acc_zero();
#pragma unroll 1
    for (int b = 0; b < 6; b++) {   // x: u_(4b-1)^7
        uint64_t u[4];
        t.finish();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[16];
            tc::ld16(t.tmem + 32 * (b & 3) + 16 * h, v);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = 2 * h + e;
                if (b == 5 && j == 3) {
                    u[3] = 0;
                    break;
                }
                if (j > 0) x = p2_seventh_and(u[j - 1], d_p2_near.own[b][j - 1], missed);
                p2_add_bytes(x, v + 8 * e);
                if (j == 2) gl::acc_mul(x, d_p2_near.far[b][0], u[0]);
                if (j == 3) {
                    gl::acc_mul(x, d_p2_near.far[b][1], u[0]);
                    gl::acc_mul(x, d_p2_near.far[b][2], u[1]);
                }
                u[j] = p2_reduce(x, missed);
            }
            t.put((b < 4 ? 4 + 2 * b : 2 * (b - 4)) + h, u[2 * h], u[2 * h + 1]);
        }
        t.meet();
        if (t.row == 0 && !*t.failed) {
            if (b == 0) t.add<4>(4, 32);
            if (b == 1) t.add<5>(6, 64);
            if (b == 2) t.add<6>(8, 96);
            if (b == 3) {
                t.begin(true);
                t.add<2>(0, 0);
                t.add<3>(2, 0);
                t.add<7>(4, 0);
                t.add<8>(6, 0);
                t.add<9>(8, 0);
                t.add<10>(10, 0);
            }
            if (b == 4) t.add<11>(0, 32);
            if (b == 5) t.add<12>(2, 48);
            t.issued.commit_to(t.done, t.turn);
        }
        if (b < 5) x = p2_seventh(u[3], missed);   // while the MMAs run
        else s[0] = u[2];
    }
    t.finish();
#pragma unroll
    for (int h = 0; h < 4; h++) {
        uint32_t v[16];
        tc::ld16(t.tmem + 48 + 16 * h, v);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            if (h == 0 && e == 0) continue;
            gl::Acc w = gl::acc_zero();
            p2_add_bytes(w, v + 8 * e);
            s[2 * h + e] = p2_reduce(w, missed);
        }
    }
    tc::fence_before();   // the next turn's first MMAs come after a barrier
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
        gl::p2t::external_linear(s, r + 1, missed);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = gl::p2t::sbox7(s[i], missed);
    p2_internal_rounds(t, s, missed);
#pragma unroll 1
    for (int r = 4; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = gl::p2t::sbox7(s[i], missed);
        gl::p2t::external_linear(s, r + 1, missed);
    }
    return !missed.any(3) && !*t.failed;   // R: at most three products and the bytes
}

}  // namespace mk
}  // namespace mb
