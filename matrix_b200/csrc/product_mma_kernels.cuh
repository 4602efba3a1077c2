// Two rounds of a sumcheck over a product of three tables per pass, with the fold and the sums on the tensor cores
// (pair_mma_kernels.cuh has the two contractions). For sum_x f(x) g(x) h(x) the next two rounds need
//     T[p][k] = sum_y (f g)(p, y) h(k, y),       k in {0, 1}^2, p in {0, 1, inf}^2,
// f g as a polynomial in the two variables: its values and leading coefficients, nine products where the pairs (i, j) of
// folded elements would be sixteen. The products are what is left on the integer pipes: 2.25 an element for both rounds
// (about 180 cycles a warp each, and 55 for the differences), where a round per pass took a fold of three tables and six to
// eight products a pair of elements (1500 instructions). Three extension tables of 2^22: first two rounds 97 us, the
// next two 65 us.
//
// Twenty-four worker warps, and one that issues the MMAs. The workers are four groups of six warps (after a fold two of twelve)
// that take the tiles in turn, each with its own buffers: a group copies, folds and multiplies its tile and meets the others
// at the issuing warp only. A thread forms the three products of one y and one p(second variable), the same for its warp. (All
// warps on every tile, two tiles in flight: 113 and 72 us, half of the issue slots waiting for the slowest warp of a tile.)
// Waits as in pair_mma_kernels.cuh.
#pragma once
#include "pair_mma_kernels.cuh"

namespace mb {
namespace pr {

constexpr int TRI_WORKERS = 768;
constexpr int TRI_BLK = TRI_WORKERS + 32;
constexpr int TRI_ENTRIES = 36;            // T[p][k] at 4 p + k, p = 3 p(second variable) + p(first), 2: inf
constexpr uint32_t TRI_TMEM = 512;
constexpr int TRI_Y = 64;                  // y of a tile
constexpr int TRI_MOST = 32768 / TRI_Y;    // tiles a block: the 32-bit sums of 2^15 rows

struct TriArgs {
    const uint64_t* in;   // three tables of 2^v elements, or 2^(v + 2) where there are challenges to fold: the two of the pass before
    size_t stride;        // words from one table to the next
    uint64_t* out;        // [3][2^v][2] folded tables, or null
    int v;                // variables left after the fold, at least 8
    uint64_t* acc;        // grid_words(TRI_ENTRIES)
    uint64_t* sums;       // pinned: [TRI_ENTRIES][2]
    uint64_t* error;      // pinned, set to 1 when a wait ran out
};

// a group's shared memory: f, g (swizzled rows of 128 bytes), h (rows of 128 bytes a y, half used) and the products (two such
// rows a y, the second for the ninth); without a fold f, g, h twice, with it the input's rows
constexpr uint32_t TRI_FG = 4096, TRI_H = 8192, TRI_P = 16384, TRI_TILE = 2 * TRI_FG + TRI_H, TRI_IN = 3 * 16384;
constexpr uint32_t TRI_RAW_GROUP = 2 * TRI_TILE + TRI_P, TRI_FOLD_GROUP = TRI_IN + TRI_TILE + TRI_P;
constexpr uint32_t TRI_RAW_SMEM = 4 * TRI_RAW_GROUP + 1024, TRI_FOLD_SMEM = 2 * TRI_FOLD_GROUP + 8192 + 1024;

// element e (of four) of y in rows of 128 bytes
template <class F, bool BASE>
__device__ __forceinline__ typename F::E2 tri_load(const uint8_t* t, uint32_t y, uint32_t e) {
    const uint32_t x = 4 * y + e;
    if constexpr (BASE) return typename F::E2{*reinterpret_cast<const uint64_t*>(t + tc::swz(x >> 4, (x >> 1) & 7) + 8 * (x & 1)), 0};
    else return load2<typename F::E2>(reinterpret_cast<const uint64_t*>(t + tc::swz(x >> 3, x & 7)));
}
// the values at p(first variable) = 0, 1, inf of the bilinear polynomial with the four elements of y, at p(second) = p1;
// CANON: the elements are canonical
template <class F, bool BASE, bool CANON>
__device__ __forceinline__ void tri_points(const uint8_t* t, uint32_t y, uint32_t p1, typename F::E2 (&v)[3]) {
    using E2 = typename F::E2;
    const auto sub = [](E2 a, E2 b) {
        if constexpr (CANON) return E2{MmaField<F>::sub_c(a.c0, b.c0), MmaField<F>::sub_c(a.c1, b.c1)};
        else return F::sub(a, b);
    };
    if (p1 < 2) {
        v[0] = tri_load<F, BASE>(t, y, 2 * p1);
        v[1] = tri_load<F, BASE>(t, y, 2 * p1 + 1);
        v[2] = sub(v[1], v[0]);
    } else {
        v[0] = sub(tri_load<F, BASE>(t, y, 2), tri_load<F, BASE>(t, y, 0));
        v[1] = sub(tri_load<F, BASE>(t, y, 3), tri_load<F, BASE>(t, y, 1));
        v[2] = F::sub(v[1], v[0]);
    }
}

template <class F, bool FOLD, bool BASE>
__global__ void __launch_bounds__(TRI_BLK, 1)
tri_mma_kernel(const TriArgs a, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr bool WORDS = BASE && !FOLD;      // the products are of words of the base field
    constexpr int C = WORDS ? 1 : 2;           // components
    constexpr int N = WORDS ? 80 : 144;        // 9 x 8 C columns, a multiple of 16
    constexpr int GROUPS = FOLD ? 2 : 4, GROUP = TRI_WORKERS / GROUPS;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t r_sm[8 * 18];
    __shared__ __align__(8) uint64_t full[GROUPS], summed[GROUPS], folded[GROUPS];   // the group is through with its tile; MMAs done
    __shared__ uint32_t tmem_sm;
    __shared__ bool last_sm;
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sm32 = tc::smem_u32(sm);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const size_t n = (size_t)1 << a.v, tiles = n / (4 * TRI_Y), per = (tiles + gridDim.x - 1) / gridDim.x;
    const size_t begin = per * blockIdx.x < tiles ? per * blockIdx.x : tiles;
    const int count = (int)((begin + per < tiles ? begin + per : tiles) - begin);   // at most TRI_MOST

    if (t == 0) {
        for (int i = 0; i < GROUPS; i++) {
            tc::mbar_init(&full[i], GROUP / 32);
            tc::mbar_init(&summed[i], 1);
            tc::mbar_init(&folded[i], 1);
        }
        tc::mbar_init_fence();
    }
    if (warp == TRI_WORKERS / 32) tc::tmem_alloc(&tmem_sm, TRI_TMEM);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_sm;
    bool failed = false;
    const auto wait = [&](uint64_t& bar, int turn) {   // the turn-th phase of a group's barrier
        if (!failed && !tc::mbar_wait(tc::smem_u32(&bar), (uint32_t)(turn & 1))) failed = true;
    };
    const auto arrive = [&](uint64_t& bar) {
        tc::fence_operands();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(tc::smem_u32(&bar));
    };
    // the products at p1 of y, from f and g in shared memory to their places in the operand
    const auto products = [&](const uint8_t* f, uint8_t* op, uint32_t y, uint32_t p1) {
        E2 x[3], z[3];
        tri_points<F, WORDS, FOLD>(f, y, p1, x);
        tri_points<F, WORDS, FOLD>(f + TRI_FG, y, p1, z);
#pragma unroll
        for (uint32_t p0 = 0; p0 < 3; p0++) {
            const uint32_t p = 3 * p1 + p0;
            if constexpr (WORDS) {
                *reinterpret_cast<uint64_t*>(op + tc::swz(y, p >> 1) + 8 * (p & 1)) = MmaField<F>::mul(x[p0].c0, z[p0].c0);
            } else {
                const E2 e = F::fma(typename F::Pre{z[p0].c0, z[p0].c1, F::times_w(z[p0].c1)}, x[p0], E2{0, 0});
                *reinterpret_cast<ulonglong2*>(op + (p >> 3) * (TRI_P / 2) + tc::swz(y, p & 7)) = make_ulonglong2(e.c0, e.c1);
            }
        }
    };
    tc::Issued issued;
    const auto issue_sums = [&](int i, uint32_t h, uint32_t op) {   // the issuing thread
        constexpr uint32_t idesc = tc::idesc_u8(N, true);
#pragma unroll
        for (int ks = 0; ks < TRI_Y / 32; ks++)
            tc::mma_i8(tmem, tc::desc_sw128(h + 4096 * ks, TRI_P / 2), tc::desc_sw128(op + 4096 * ks, TRI_P / 2), idesc, !(i == 0 && ks == 0));
        issued.commit_to(tc::smem_u32(&summed[i % GROUPS]), i / GROUPS);
    };
    const int group = t / GROUP, gt = t % GROUP, gw = gt >> 5;   // a worker's group, its thread and warp in it

    if constexpr (!FOLD) {
        constexpr uint32_t UNITS = BASE ? 128 : 256, PER = BASE ? 2 : 4;   // 16-byte units of a table, of a y
        if (t < TRI_WORKERS) {
            const uint32_t off = group * TRI_RAW_GROUP;
            const auto load = [&](int turn) {
                const int i = group + GROUPS * turn;
                if (i < count && !failed) {
                    const uint32_t dst = sm32 + off + (turn & 1) * TRI_TILE;
                    const uint64_t* src = a.in + (begin + i) * (size_t)(2 * UNITS);
                    for (uint32_t c = gt; c < 3 * UNITS; c += GROUP) {
                        const uint32_t k = c / UNITS, u = c % UNITS;
                        tc::copy16(dst + k * TRI_FG + (k < 2 ? tc::swz(u >> 3, u & 7) : tc::swz(u / PER, u % PER)), src + a.stride * k + 2 * u);
                    }
                }
                tc::copy_commit();
            };
            load(0);
            for (int turn = 0; group + GROUPS * turn < count; turn++) {
                tc::copy_wait<0>();
                tc::fence_operands();
                tc::named_sync(GROUP, 1 + group);          // the whole tile is here
                if (turn > 0) wait(summed[group], turn - 1);   // the other buffer and the products' are free
                load(turn + 1);
                if (!failed) products(sm + off + (turn & 1) * TRI_TILE, sm + off + 2 * TRI_TILE, 32 * (gw & 1) + lane, gw >> 1);
                arrive(full[group]);
            }
        } else if (lane == 0) {
            for (int i = 0; i < count; i++) {
                const int g = i % GROUPS, turn = i / GROUPS;
                wait(full[g], turn);
                if (failed) break;
                tc::fence_after();
                const uint32_t off = sm32 + g * TRI_RAW_GROUP;
                issue_sums(i, off + (turn & 1) * TRI_TILE + 2 * TRI_FG, off + 2 * TRI_TILE);
            }
            issued.drain();
        }
    } else {
        constexpr int le = BASE ? 2 : 1;                           // log2 of the folded elements in 128 bytes of input
        constexpr uint32_t rows = 256u >> le, units = 8 * rows;    // of a table
        constexpr uint32_t cst = GROUPS * TRI_FOLD_GROUP, fold_cols = 256;   // 128 columns a group
        constexpr uint32_t idesc_f = tc::idesc_u8(16 << le, false);
        const auto load = [&](int turn) {
            const int i = group + GROUPS * turn;
            if (i < count && !failed) {
                const uint32_t dst = sm32 + group * TRI_FOLD_GROUP;
                const uint64_t* src = a.in + (begin + i) * (size_t)(2 * units);
                for (uint32_t c = gt; c < units; c += GROUP)
#pragma unroll
                    for (uint32_t k = 0; k < 3; k++)
                        tc::copy16(dst + k * rows * 128 + tc::swz(c >> 3, c & 7), src + a.stride * k + 2 * c);
            }
            tc::copy_commit();
        };
        if (t < TRI_WORKERS) {
            load(0);
            fold_operand<F, BASE>(sm + cst, le, fw, TRI_WORKERS);
            tc::copy_wait<0>();
            tc::fence_operands();
        }
        __syncthreads();
        if (t < TRI_WORKERS) {
            uint8_t* buf = sm + group * TRI_FOLD_GROUP + TRI_IN;   // f, g, h, products
            const uint32_t lr = (gw & 3) * 32 + lane;
            for (int turn = 0; group + GROUPS * turn < count; turn++) {
                const size_t tile = begin + group + GROUPS * turn;
                wait(folded[group], turn);
                tc::fence_after();
                load(turn + 1);   // the tile's MMAs have read the input
                if (turn > 0) wait(summed[group], turn - 1);
                // 128 rows and one element of each a unit: three tables of 128 rows (le = 1), or of 64 (le = 2)
                for (uint32_t u = gw >> 2; u < (le == 1 ? 6u : 8u); u += GROUP / 128) {
                    const uint32_t row = (u >> le) * 128 + lr, k = row / rows, x = ((row % rows) << le) + (u & ((1u << le) - 1));
                    if (k >= 3) continue;   // a warp's rows are one table's
                    uint32_t s[16];
                    tc::ld16(tmem + ((uint32_t)(32 * (gw & 3)) << 16) + fold_cols + group * 128 + u * 16, s);
                    const E2 e{bytes_value<F>(s), bytes_value<F>(s + 8)};
                    if (failed) continue;
                    if (a.out != nullptr) store2(a.out + 2 * (n * k + tile * (size_t)(4 * TRI_Y) + x), e.c0, e.c1);
                    uint8_t* dst = buf + k * TRI_FG + (k < 2 ? tc::swz(x >> 3, x & 7) : tc::swz(x >> 2, x & 3));
                    *reinterpret_cast<ulonglong2*>(dst) = make_ulonglong2(e.c0, e.c1);
                }
                tc::named_sync(GROUP, 1 + group);
                if (gw / 6 == (turn & 1)) {   // 192 threads' worth of products
                    const uint32_t w = gw % 6;
                    if (!failed) products(buf, buf + TRI_TILE, 32 * (w & 1) + lane, w >> 1);
                }
                tc::copy_wait<0>();   // the next tile
                arrive(full[group]);
            }
        } else if (lane == 0) {
            const auto issue_fold = [&](int i) {
                const uint32_t g = i % GROUPS, st = sm32 + g * TRI_FOLD_GROUP;
                for (uint32_t q = 0; q < (le == 1 ? 3u : 2u); q++)
                    for (uint32_t ks = 0; ks < 4; ks++)
                        tc::mma_i8(tmem + fold_cols + g * 128 + q * (16u << le), tc::desc_sw128(st + q * 16384 + ks * 32, 0),
                                   tc::desc_sw128(sm32 + cst + ks * 32, 0), idesc_f, ks > 0);
                issued.commit_to(tc::smem_u32(&folded[g]), i / GROUPS);
            };
            tc::fence_after();
            for (int i = 0; i < GROUPS && i < count; i++) issue_fold(i);
            for (int i = 0; i < count; i++) {
                wait(full[i % GROUPS], i / GROUPS);
                if (failed) break;
                tc::fence_after();
                const uint32_t buf = sm32 + (i % GROUPS) * TRI_FOLD_GROUP + TRI_IN;
                if (i + GROUPS < count) issue_fold(i + GROUPS);
                issue_sums(i, buf + 2 * TRI_FG, buf + TRI_TILE);
            }
            issued.drain();
        }
    }
    tc::copy_wait<0>();
    __syncwarp();
    // every tile's MMAs: the last of each group
    if (t < GROUPS && t < count) wait(summed[t], (count - 1 - t) / GROUPS);
    tc::fence_before();
    failed = __syncthreads_or(failed);
    tc::fence_after();
    if (count > 0 && !failed && t < TRI_WORKERS && (warp & 3) < C) {   // lanes: byte of h(k); columns: byte of the product p
        const int q = warp & 3;
        const uint64_t scale = 1ULL << (8 * (lane & 7));
        for (int ga = warp >> 2; ga < 9 * C; ga += TRI_WORKERS / 128) {
            const uint64_t v = gather_word<F>(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(8 * ga), scale);
            if ((lane & 7) == 0) r_sm[(4 * q + (lane >> 3)) * 18 + ga] = v;
        }
        tc::fence_before();
    }
    __syncthreads();
    if (warp == TRI_WORKERS / 32) tc::tmem_free(tmem, TRI_TMEM);
    if (failed) {
        if (t == 0) *a.error = 1;
        return;
    }
    E2 sum{0, 0};
    if (t < TRI_ENTRIES && count > 0) {
        const uint64_t* r = r_sm + (t & 3) * C * 18 + (t >> 2) * C;   // [component of h][component of the product]
        if constexpr (WORDS) sum = E2{F::canon(r[0]), 0};
        else sum = E2{F::canon(MmaField<F>::add(r[0], F::times_w(r[19]))), F::canon(MmaField<F>::add(r[1], r[18]))};
    }
    if (gridDim.x > 1) {
        if (t < TRI_ENTRIES) grid_add(a.acc, TRI_ENTRIES, blockIdx.x, t, sum.c0, sum.c1);
        if (!grid_last(a.acc, &last_sm, gridDim.x)) return;
        if (t < TRI_ENTRIES) sum = grid_take<F>(a.acc, TRI_ENTRIES, t);
    }
    if (t < TRI_ENTRIES) store2(a.sums + 2 * t, sum.c0, sum.c1);
}

}  // namespace pr
}  // namespace mb
