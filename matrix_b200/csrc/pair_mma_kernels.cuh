// The pass of pair_kernels.cuh on the tensor cores, for tables of a thousand elements and more.
//
// Both of its halves are contractions of exact integers, and a 64-bit word is eight unsigned bytes as it lies in memory:
//   fold   sum_m e_m t(m + 2^F y): a row of an operand is 128 bytes of the input, the other operand holds the bytes of
//          2^(8 i) e_m mod p for input byte i, so eight 32-bit sums per component come back, sum_k S_k 2^(8 k), S_k < 2^23;
//   sums   M[i][j] = sum_y w(y) a(i + G y) b(j + G y): rows y of 128 bytes (eight extension elements, sixteen words of the
//          base field), contracted over y as they lie (both operands MN-major): all 128 x 128 (x 256) byte products, whose
//          sums over 2^15 rows stay below 2^31; once per 2^15 rows or weight of WH they are put together to field elements.
// A product of extension elements on the integer pipes takes four chains of 24 cycles a warp (64 x 64 into a 160-bit sum);
// here 256 rows' worth of them costs the tensor pipe 64 cycles an SM, so what is left is the traffic, the weights (a is
// multiplied by WL before it becomes an operand) and the reductions after a fold (about 30 instructions a component).
// Sixteen instances of 2^22 under a weight: first pass 740 -> 268 us, the pass that folds it 672 -> 240 us.
//
// One block an SM: sixteen warps that copy, weigh and reduce, and one that issues the MMAs. They meet at mbarriers only, so a
// warp may be two tiles ahead of another. Copies to shared memory run two or more tiles ahead (cp.async into the swizzled
// operand layout), the fold's MMAs two tiles ahead of the warps that reduce them. Every wait is bounded; a thread whose wait
// ran out goes on without waiting or touching buffers (the block's barriers count every warp), and the block sets *a.error
// (tcgen05.cuh).
#pragma once
#include "pair_kernels.cuh"
#include "tcgen05.cuh"

namespace mb {
namespace pr {

constexpr int MMA_WORKERS = 512;
constexpr int MMA_BLK = MMA_WORKERS + 32;
constexpr int MMA_ROW_BITS = 14;           // variables of WL
constexpr uint32_t MMA_TMEM = 256;
constexpr int MMA_RAW_ROWS = 128;          // rows of a tile without a fold
constexpr int MMA_FOLD_TILE = 256;         // folded elements of a tile
constexpr uint32_t MMA_HALF = MMA_RAW_ROWS * 128;

// log2 of the fewest elements after the fold; input bytes of a folded element from 32 to 128
constexpr int mma_min_vars(bool fold, bool base) { return fold ? 8 : base ? 11 : 10; }
// (a block of one round is a proof's last: no pass folds one challenge)
constexpr bool mma_folds(int fb, bool base) { return fb >= 2 && fb <= (base ? 4 : 3); }

struct PairMmaArgs {
    int fb;                   // challenges to fold (0: none)
    const uint64_t *a, *b;    // as PairArgs
    size_t in_stride;
    uint64_t* out;
    int v;                    // variables left after the fold
    int g;                    // rounds of the next block: 1 .. 3, with base words and no fold up to 4
    int lo;                   // weighted passes: variables of WL
    int row_shift;            // log2 of the elements between two entries of WH (63: WH is a single 1)
    size_t row_mask;
    const uint64_t *wl, *wh;
    uint64_t* acc;            // [instance][grid_words(4^g)]
    uint64_t* sums;           // pinned: [instance][4^g][2]
    uint64_t* error;          // pinned, set to 1 when a wait ran out
};

template <class F> struct MmaField;
template <> struct MmaField<GlF> {
    static __device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) { return gl::mul(a, b); }
    static __device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) { return gl::add(a, b); }
    static __device__ __forceinline__ uint64_t sub_c(uint64_t a, uint64_t b) { return gl::sub_c(a, b); }   // b canonical
    static __device__ __forceinline__ uint64_t red128(uint64_t lo, uint64_t hi) { return gl::reduce128(lo, hi); }
    // lo + hi 2^64 for hi < 2^18
    static __device__ __forceinline__ uint64_t red_small(uint64_t lo, uint32_t hi) {
        uint32_t c;
        const uint64_t s = gl::add_carry(lo, ((uint64_t)hi << 32) - hi, c);
        return s + (uint64_t)(0u - c);
    }
};
template <> struct MmaField<AglF> {
    static __device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) { return agl::mul(a, b); }
    static __device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) { return agl::add(a, b); }
    static __device__ __forceinline__ uint64_t sub_c(uint64_t a, uint64_t b) { return agl::sub_c(a, b); }   // b canonical
    static __device__ __forceinline__ uint64_t red128(uint64_t lo, uint64_t hi) { return agl::reduce128(lo, hi); }
    static __device__ __forceinline__ uint64_t red_small(uint64_t lo, uint32_t hi) {
        uint32_t c;
        const uint64_t s = gl::add_carry(lo, ((uint64_t)hi << 32) + hi * 31u, c);
        return s + gl::pack64(c * 31u, c);
    }
};

// sum_k s[k] 2^(8 k) mod p for s[k] <= 255^2 * 128: the words at distance four lie side by side
template <class F>
__device__ __forceinline__ uint64_t bytes_value(const uint32_t* s) {
    const uint64_t u = gl::pack64(s[0], s[4]) + (gl::pack64(s[1], s[5]) << 8), w = gl::pack64(s[2], s[6]) + (gl::pack64(s[3], s[7]) << 8);
    uint32_t c;
    const uint64_t lo = gl::add_carry(u, w << 16, c);
    return F::canon(MmaField<F>::red_small(lo, (uint32_t)(w >> 48) + c));
}
// the same for any 32-bit s[k], loose
template <class F>
__device__ __forceinline__ uint64_t bytes_value_wide(const uint32_t* s) {
    unsigned __int128 x = gl::pack64(s[0], s[4]);
    x += (unsigned __int128)gl::pack64(s[1], s[5]) << 8;
    x += (unsigned __int128)gl::pack64(s[2], s[6]) << 16;
    x += (unsigned __int128)gl::pack64(s[3], s[7]) << 24;
    return MmaField<F>::red128((uint64_t)x, (uint64_t)(x >> 64));
}

// w(y) x for an element of the base field (BASE) or the extension
template <class F, bool BASE>
__device__ __forceinline__ typename F::E2 weigh(const typename F::Pre& w, uint64_t c0, uint64_t c1) {
    if constexpr (BASE) return typename F::E2{MmaField<F>::mul(w.c0, c0), MmaField<F>::mul(w.c1, c0)};
    else return F::fma(w, typename F::E2{c0, c1}, typename F::E2{0, 0});
}

// The fold's operand of weights, K-major, by the first `workers` threads: row (sub, component, byte) holds that byte of the
// factor of each input byte, and zero outside the sub-th of the 2^le elements in 128 bytes of input.
template <class F, bool BASE>
__device__ __forceinline__ void fold_operand(uint8_t* cst, int le, const FoldWeights<F>& fw, uint32_t workers) {
    const uint32_t t = threadIdx.x, words = 16u >> le;   // words of one element
    for (uint32_t x = t; x < (16u << le) * 8; x += workers) *reinterpret_cast<uint4*>(cst + 16 * x) = make_uint4(0, 0, 0, 0);
    tc::named_sync(workers);
    for (uint32_t x = t; x < words * 16; x += workers) {
        const uint32_t comp = x & 1, i = (x >> 1) & 7, w = x >> 4;
        uint64_t f;
        if constexpr (BASE) {
            f = comp ? fw.w[w].c1 : fw.w[w].c0;
        } else {
            const typename F::Pre& e = fw.w[w >> 1];
            f = comp ? ((w & 1) ? e.c0 : e.c1) : ((w & 1) ? e.c1w : e.c0);
        }
        f = F::canon(MmaField<F>::mul(f, 1ULL << (8 * i)));
        for (uint32_t sub = 0; sub < (1u << le); sub++) {
            const uint32_t col = sub * 8 * words + 8 * w + i;
            for (uint32_t byte = 0; byte < 8; byte++) {
                const uint32_t row = sub * 16 + comp * 8 + byte;
                cst[tc::swz(row, col >> 4) + (col & 15)] = (uint8_t)(f >> (8 * byte));
            }
        }
    }
}
// one group of eight columns of the accumulators: byte products of two words, by the lane's byte of the other operand; the
// sum over its eight lanes, loose, in each of them
template <class F>
__device__ __forceinline__ uint64_t gather_word(uint32_t addr, uint64_t scale) {
    using M = MmaField<F>;
    uint32_t s[8];
    tc::ld8(addr, s);
    uint64_t v = M::mul(bytes_value_wide<F>(s), scale);
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) v = M::add(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// Sums of the block's rows of 4^g byte products: what the accumulators hold, put together by byte of b (eight lanes), byte
// of a (eight columns), component and diagonal block (rows hold more elements than 2^g when the block is shorter).
// r_sm: 16 x 32 words. Threads below 4^g get the entry M[t >> g][t mod 2^g].
// A: components of an element of a; B: of b. The accumulators start at tensor-memory column 0.
template <class F, int A, int B>
__device__ __forceinline__ typename F::E2 gather_sums(uint32_t tmem, uint64_t* r_sm, int g) {
    using E2 = typename F::E2;
    using M = MmaField<F>;
    constexpr int ELEMS = B == 1 ? 16 : 8;               // elements of a row
    constexpr int GROUPS_A = ELEMS * A;                  // groups of eight columns
    const int t = threadIdx.x, lane = t & 31, q = (t >> 5) & 3, part = t >> 7;
    const uint64_t scale = 1ULL << (8 * (lane & 7));
#pragma unroll
    for (int x = 0; x < GROUPS_A / 4; x++) {
        const int ga = part * (GROUPS_A / 4) + x;
        const uint64_t v = gather_word<F>(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(8 * ga), scale);
        if ((lane & 7) == 0) r_sm[(4 * q + (lane >> 3)) * 32 + ga] = v;
    }
    tc::fence_before();
    tc::named_sync(MMA_WORKERS);
    E2 e{0, 0};
    const int side = 1 << g;
    if (t < side * side) {
        const int i = t >> g, j = t & (side - 1);
        for (int d = 0; d < ELEMS; d += side) {
            const uint64_t* rj = r_sm + (j + d) * B * 32 + (i + d) * A;   // [component of b][component of a]
            uint64_t c0 = rj[0], c1 = 0;
            if constexpr (A == 2) c1 = rj[1];
            if constexpr (B == 2) {
                c0 = M::add(c0, F::times_w(rj[33]));
                c1 = M::add(c1, rj[32]);
            }
            e = F::add(e, E2{c0, c1});
        }
    }
    return e;
}

constexpr int MMA_FOLD_STAGES = 3;
__host__ __device__ constexpr uint32_t mma_fold_stage(int log_epr) { return 65536u >> log_epr; }
// dynamic shared memory, with 1024 bytes to align it
__host__ __device__ constexpr uint32_t mma_fold_smem(int log_epr) { return MMA_FOLD_STAGES * mma_fold_stage(log_epr) + 16384 + 8192 + 1024; }
__host__ __device__ constexpr int mma_raw_stages(bool weighted) { return weighted ? 4 : 6; }
__host__ __device__ constexpr uint32_t mma_raw_smem(bool base, bool weighted) {
    return mma_raw_stages(weighted) * 2 * MMA_HALF + (weighted ? (base ? 4 : 2) * MMA_HALF : 0) + 1024;
}

// FOLD: there are challenges to fold. BASE: input words of the base field. Grid (blocks, instances).
template <class F, bool FOLD, bool BASE, bool WEIGHTED>
__global__ void __launch_bounds__(MMA_BLK, 1)
pair_mma_kernel(const PairMmaArgs a, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr int CA = (FOLD || !BASE || WEIGHTED) ? 2 : 1, CB = (FOLD || !BASE) ? 2 : 1;   // components of a, b as operands
    constexpr int N = (CB == 1 ? 16 : 8) * CA * 8;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t r_sm[16 * 32];
    __shared__ __align__(8) uint64_t full[2], summed[2], folded[2];   // by tile mod 2: every warp is through, the MMAs are done
    __shared__ uint32_t tmem_sm;
    __shared__ bool last_sm;
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sm32 = tc::smem_u32(sm);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, k = blockIdx.y;
    const uint64_t *pa = a.a + a.in_stride * k, *pb = a.b + a.in_stride * k;
    const size_t n = (size_t)1 << a.v;
    constexpr int TILE = FOLD ? MMA_FOLD_TILE : MMA_RAW_ROWS * (BASE ? 16 : 8);   // elements a table
    const size_t tiles = n / TILE, per = (tiles + gridDim.x - 1) / gridDim.x, first = per * blockIdx.x < tiles ? per * blockIdx.x : tiles;
    const int count = (int)((first + per < tiles ? first + per : tiles) - first);
    // tiles between two readings of the accumulators: 2^15 rows at most, and a row of WL where WH has more than one entry
    const size_t cap = FOLD ? 1024 : 256;
    const size_t flush = WEIGHTED && a.row_shift < 63 && ((size_t)1 << a.row_shift) / TILE < cap ? ((size_t)1 << a.row_shift) / TILE : cap;

    if (t == 0) {
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&full[i], MMA_WORKERS / 32);
            tc::mbar_init(&summed[i], 1);
            tc::mbar_init(&folded[i], 1);
        }
        tc::mbar_init_fence();
    }
    if (warp == MMA_WORKERS / 32) tc::tmem_alloc(&tmem_sm, MMA_TMEM);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_sm;
    bool failed = false;
    // waits for phase n of a barrier whose phases alternate between two
    const auto wait = [&](uint64_t* bar, int n) {
        if (!failed && !tc::mbar_wait(tc::smem_u32(&bar[n & 1]), (uint32_t)((n >> 1) & 1))) failed = true;
    };
    const auto arrive = [&](int n) {   // a warp is through with tile n
        tc::fence_operands();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(tc::smem_u32(&full[n & 1]));
    };
    const auto starts = [&](int i) { return i == 0 || (first + i) % flush == 0; };   // the accumulators start at tile i
    E2 sum{0, 0};
    const auto take_sums = [&](int i) {   // after tile i where the accumulators end
        if (!((first + i + 1) % flush == 0 || i + 1 == count)) return;
        wait(summed, i);
        tc::fence_after();
        const E2 e = gather_sums<F, CA, CB>(tmem, r_sm, a.g);
        if (t < (1 << (2 * a.g))) {
            if constexpr (WEIGHTED) {
                const size_t row = a.row_shift < 63 ? (((first + i) * TILE) >> a.row_shift) & a.row_mask : 0;
                sum = F::fma(load_weight<F>(a.wh + 4 * row), e, sum);
            } else {
                sum = F::add(sum, e);
            }
        }
    };
    const auto weight = [&](size_t x) {   // of element x; W c1 only where it is used
        const uint64_t* p = a.wl + 4 * ((x >> a.g) & (((size_t)1 << a.lo) - 1));
        if constexpr (FOLD || !BASE) return load_weight<F>(p);
        const E2 w = load2<E2>(p);
        return typename F::Pre{w.c0, w.c1, 0};
    };
    constexpr uint32_t idesc_s = tc::idesc_u8(N, true);

    if constexpr (!FOLD) {
        constexpr int NS = mma_raw_stages(WEIGHTED);
        constexpr uint32_t STAGE = 2 * MMA_HALF;   // b, then a
        constexpr uint32_t abuf = NS * STAGE;      // weighted a: two buffers of one half (extension: eight elements a row) or two
        constexpr uint32_t ABUF = (BASE ? 2 : 1) * MMA_HALF;
        if (t < MMA_WORKERS) {
            const auto load = [&](int i) {
                if (i < count && !failed) {
                    const uint32_t dst = sm32 + (uint32_t)(i % NS) * STAGE;
                    const size_t w = (first + i) * (size_t)(MMA_HALF / 8);
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        const uint32_t c = t + x * MMA_WORKERS, off = tc::swz(c >> 3, c & 7);
                        tc::copy16(dst + off, pb + w + 2 * c);
                        tc::copy16(dst + MMA_HALF + off, pa + w + 2 * c);
                    }
                }
                tc::copy_commit();
            };
            for (int i = 0; i < NS - 2; i++) load(i);
            for (int i = 0; i < count; i++) {
                typename F::Pre w[2];
                if constexpr (WEIGHTED) {
#pragma unroll
                    for (int x = 0; x < 2; x++) w[x] = weight((first + i) * TILE + (BASE ? 2 : 1) * (size_t)(t + x * MMA_WORKERS));
                }
                if (i >= 2) wait(summed, i - 2);   // its stage and its buffer are free
                load(i + NS - 2);
                tc::copy_wait<NS - 2>();
                if constexpr (WEIGHTED) {
                    const uint8_t* src = sm + (uint32_t)(i % NS) * STAGE + MMA_HALF;
                    uint8_t* dst = sm + abuf + (i & 1) * ABUF;
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        const uint32_t c = t + x * MMA_WORKERS, r = c >> 3, u = c & 7;   // the units this thread copied itself
                        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(src + tc::swz(r, u));
                        if constexpr (BASE) {
                            const E2 e0 = weigh<F, true>(w[x], p.x, 0), e1 = weigh<F, true>(w[x], p.y, 0);
                            uint8_t* half = dst + (u >> 2) * MMA_HALF;
                            if (!failed) {
                                *reinterpret_cast<ulonglong2*>(half + tc::swz(r, 2 * (u & 3))) = make_ulonglong2(e0.c0, e0.c1);
                                *reinterpret_cast<ulonglong2*>(half + tc::swz(r, 2 * (u & 3) + 1)) = make_ulonglong2(e1.c0, e1.c1);
                            }
                        } else {
                            const E2 e = weigh<F, false>(w[x], p.x, p.y);
                            if (!failed) *reinterpret_cast<ulonglong2*>(dst + tc::swz(r, u)) = make_ulonglong2(e.c0, e.c1);
                        }
                    }
                }
                arrive(i);
                take_sums(i);
            }
        } else if (lane == 0) {
            tc::Issued issued;
            for (int i = 0; i < count && !failed; i++) {
                wait(full, i);
                if (failed) break;
                tc::fence_after();
                const uint32_t st = sm32 + (uint32_t)(i % NS) * STAGE, opa = WEIGHTED ? sm32 + abuf + (i & 1) * ABUF : st + MMA_HALF;
                const bool start = starts(i);
#pragma unroll
                for (int ks = 0; ks < MMA_RAW_ROWS / 32; ks++)
                    tc::mma_i8(tmem, tc::desc_sw128(st + 4096 * ks, MMA_HALF), tc::desc_sw128(opa + 4096 * ks, MMA_HALF), idesc_s,
                               !(start && ks == 0));
                issued.commit_to(tc::smem_u32(&summed[i & 1]), i >> 1);
            }
            issued.drain();
        }
    } else {
        const int le = BASE ? 4 - a.fb : 3 - a.fb;                 // log2 of the folded elements in 128 bytes of input
        const uint32_t stage = mma_fold_stage(le);
        const uint32_t ops = MMA_FOLD_STAGES * stage, cst = ops + 16384;   // sums' operands [buffer][b, a]; weights of the fold
        constexpr uint32_t fold_cols = 128;                        // two buffers of 64 columns above the sums
        const uint32_t idesc_f = tc::idesc_u8(16 << le, false);
        const auto load = [&](int i) {
            if (i < count && !failed) {
                const uint32_t dst = sm32 + (uint32_t)(i % MMA_FOLD_STAGES) * stage, rows = 256u >> le;
                const size_t w = (first + i) * (size_t)(rows * 16);
                for (uint32_t c = t; c < 8 * rows; c += MMA_WORKERS) {
                    tc::copy16(dst + tc::swz(c >> 3, c & 7), pa + w + 2 * c);
                    tc::copy16(dst + rows * 128 + tc::swz(c >> 3, c & 7), pb + w + 2 * c);
                }
            }
            tc::copy_commit();
        };
        if (t < MMA_WORKERS) {
            for (int i = 0; i < 3; i++) load(i);
            fold_operand<F, BASE>(sm + cst, le, fw, MMA_WORKERS);
            tc::copy_wait<1>();   // tiles 0 and 1
            tc::fence_operands();
        }
        __syncthreads();
        if (t < MMA_WORKERS) {
            // this thread's element: quarter `part` of the block's warps, lane row `lr` of a group of 128 rows
            const uint32_t part = warp >> 2, lr = (warp & 3) * 32 + lane;
            uint32_t table, elem;
            if (le == 0) { table = part >> 1; elem = (part & 1) * 128 + lr; }
            else if (le == 1) { table = part >> 1; elem = 2 * lr + (part & 1); }
            else { table = lr >> 6; elem = 4 * (lr & 63) + part; }
            uint64_t* out = a.out == nullptr ? nullptr : a.out + ((size_t)4 << a.v) * k + 2 * (n * table + elem);
            uint8_t* op = sm + ops + (1 - table) * 4096 + tc::swz(elem >> 3, elem & 7);
            for (int i = 0; i < count; i++) {
                typename F::Pre w;
                if constexpr (WEIGHTED) w = weight((first + i) * MMA_FOLD_TILE + elem);
                wait(folded, i);
                tc::fence_after();
                load(i + 3);   // into the stage that tile i's MMAs have read
                uint32_t s[16];
                tc::ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + fold_cols + (i & 1) * 64 + part * 16, s);
                E2 f{bytes_value<F>(s), bytes_value<F>(s + 8)};
                if (out != nullptr && !failed) store2(out + 2 * ((first + i) * (size_t)MMA_FOLD_TILE), f.c0, f.c1);
                if constexpr (WEIGHTED) {
                    if (table == 0) f = weigh<F, false>(w, f.c0, f.c1);
                }
                if (i >= 2) wait(summed, i - 2);
                if (!failed) *reinterpret_cast<ulonglong2*>(op + (i & 1) * 8192) = make_ulonglong2(f.c0, f.c1);
                tc::copy_wait<1>();   // tile i + 2
                arrive(i);
                take_sums(i);
            }
        } else if (lane == 0) {
            tc::Issued issued;
            const auto issue_fold = [&](int i) {
                const uint32_t st = sm32 + (uint32_t)(i % MMA_FOLD_STAGES) * stage;
                for (uint32_t q = 0; q < (4u >> le); q++)
                    for (uint32_t ks = 0; ks < 4; ks++)
                        tc::mma_i8(tmem + fold_cols + (i & 1) * 64 + q * (16u << le), tc::desc_sw128(st + q * 16384 + ks * 32, 0),
                                   tc::desc_sw128(sm32 + cst + ks * 32, 0), idesc_f, ks > 0);
                issued.commit_to(tc::smem_u32(&folded[i & 1]), i >> 1);
            };
            tc::fence_after();
            for (int i = 0; i < 2 && i < count; i++) issue_fold(i);
            for (int i = 0; i < count && !failed; i++) {
                wait(full, i);   // tile i is in the operands, its sums of the fold are read, tile i + 2 is in shared memory
                if (failed) break;
                tc::fence_after();
                const uint32_t op = sm32 + ops + (i & 1) * 8192;
                tc::mma_i8(tmem, tc::desc_sw128(op, 4096), tc::desc_sw128(op + 4096, 4096), idesc_s, !starts(i));
                issued.commit_to(tc::smem_u32(&summed[i & 1]), i >> 1);
                if (i + 2 < count) issue_fold(i + 2);
            }
            issued.drain();
        }
    }
    tc::copy_wait<0>();
    __syncwarp();
    tc::fence_before();
    failed = __syncthreads_or(failed);
    if (warp == MMA_WORKERS / 32) tc::tmem_free(tmem, MMA_TMEM);
    if (failed) {
        if (t == 0) *a.error = 1;
        return;
    }
    // ---- over the blocks ----
    const int E = 1 << (2 * a.g);
    if (gridDim.x > 1) {
        uint64_t* acc = a.acc + grid_words(E) * k;
        if (t < E) grid_add(acc, E, blockIdx.x, t, F::canon(sum.c0), F::canon(sum.c1));
        if (!grid_last(acc, &last_sm, gridDim.x)) return;
        if (t < E) sum = grid_take<F>(acc, E, t);
    }
    if (t < E) store2(a.sums + 2 * ((size_t)k * E + t), F::canon(sum.c0), F::canon(sum.c1));
}

}  // namespace pr
}  // namespace mb
