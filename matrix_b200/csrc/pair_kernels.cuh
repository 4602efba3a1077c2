// Several rounds of a sumcheck over products of two tables per pass.
//
// For sum_x w(x) a(x) b(x) (w = 1, or an eq polynomial) B consecutive rounds, which bind the low B variables, need
// nothing of the tables but the 2^B x 2^B matrix
//     M[i][j] = sum_y w'(y) a(i + 2^B y) b(j + 2^B y),          w' = w over the variables above the low B,
// because folding and evaluating the round polynomials only combine rows and columns: the host runs the B rounds on
// M. One pass over the tables folds the F challenges of the block of rounds before (a dot product with their eq
// vector, reduced once), stores the folded tables and accumulates M from them. Per element that is 2^F products for
// the fold and 2^B for M, against one read and write of the tables, one launch and one synchronisation per round when
// every round has its own pass; B grows as the tables shrink (what bounds a large table is its traffic and products,
// a small one the launch).
//
// A block takes tiles of 256 folded elements per table: thread t folds element t of a and of b into shared memory,
// then thread t = (y group, i, j) adds its entry of M over the tile, 2^B products. Weights: w'(y) = WL[y mod 2^lo]
// WH[y >> lo]; a is multiplied by WL before it enters shared memory, and a thread's sum by WH whenever the row ends.
#pragma once
#include "agl_traits.cuh"

namespace mb {
namespace pr {

constexpr int BLK = 256;
constexpr int MAX_B = 4;
constexpr int ROW_BITS = 10;   // variables of WL

// ---- fields --------------------------------------------------------------------------------------
struct GlF {
    using E2 = gl::E2;
    using Pre = gl::E2Pre;
    static constexpr uint32_t W = 7;
    static __device__ __forceinline__ uint64_t canon(uint64_t x) { return gl::canon(x); }
    static __device__ __forceinline__ uint64_t red(const gl::Acc& s) { return gl::acc_reduce(s); }
    static __device__ __forceinline__ uint64_t redw(const gl::Acc& s) { return gl::acc_reduce_wide(s); }
    static __device__ __forceinline__ uint64_t times_w(uint64_t x) { return gl::mul_small(x, W); }
    static __device__ __forceinline__ E2 add(E2 a, E2 b) { return gl::e2_add(a, b); }
    static __device__ __forceinline__ E2 sub(E2 a, E2 b) { return gl::e2_sub(a, b); }
    static __device__ __forceinline__ E2 mul(E2 a, E2 b) { return gl::e2_mul_lazy(a, b); }
    static __device__ __forceinline__ E2 fma(Pre w, E2 x, E2 a) { return gl::e2_fma_pre(w, x, a); }
};
struct AglF {
    using E2 = agl::E2;
    using Pre = agl::E2Pre;
    static constexpr uint32_t W = 3;
    static __device__ __forceinline__ uint64_t canon(uint64_t x) { return agl::canon(x); }
    static __device__ __forceinline__ uint64_t red(const gl::Acc& s) { return agl::acc_reduce(s); }
    static __device__ __forceinline__ uint64_t redw(const gl::Acc& s) { return agl::acc_reduce_wide(s); }
    static __device__ __forceinline__ uint64_t times_w(uint64_t x) { return agl::mul_small(x, W); }
    static __device__ __forceinline__ E2 add(E2 a, E2 b) { return agl::e2_add(a, b); }
    static __device__ __forceinline__ E2 sub(E2 a, E2 b) { return agl::e2_sub(a, b); }
    static __device__ __forceinline__ E2 mul(E2 a, E2 b) { return agl::e2_mul_lazy(a, b); }
    static __device__ __forceinline__ E2 fma(Pre w, E2 x, E2 a) { return agl::e2_fma_pre(w, x, a); }
};
template <class E2>
__device__ __forceinline__ E2 load2(const uint64_t* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return E2{v.x, v.y};
}
__device__ __forceinline__ void store2(uint64_t* p, uint64_t c0, uint64_t c1) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(c0, c1);
}

// ---- eq tables: entries (c0, c1, W c1, 0) over variables [first, first + bits) of the point -----------
struct TableDesc {
    int first, bits;
    size_t off;   // words
};
constexpr int MAX_TABLES = 48;
constexpr int MAX_POINT = 40;
struct TableSet {
    TableDesc d[MAX_TABLES];
    uint64_t pt[2 * MAX_POINT];   // the point's coordinates, (c0, c1)
};
// A block forms the products over each seven variables of its table (a tree of six products a thread) and then its share
// of the entries from them, so a table of 2^14 takes two barriers on 64 SMs and not fourteen doublings on one.
constexpr int EQ_PART = 7, EQ_PARTS = 4;      // tables of up to 28 variables
inline unsigned eq_table_chunks(const TableSet& set, int nt) {   // blocks a table
    int bits = 0;
    for (int i = 0; i < nt; i++) bits = set.d[i].bits > bits ? set.d[i].bits : bits;
    return bits <= 8 ? 1u : bits >= 14 ? 64u : 1u << (bits - 8);
}
template <class F>
__global__ void __launch_bounds__(BLK)
eq_tables_kernel(const __grid_constant__ TableSet set, uint64_t* __restrict__ tabs) {
    using E2 = typename F::E2;
    __shared__ E2 part[EQ_PARTS][1 << EQ_PART];
    const TableDesc d = set.d[blockIdx.x];
    const size_t n = (size_t)1 << d.bits, first = (size_t)blockIdx.y * BLK;
    if (first >= n) return;
    const int parts = d.bits > 0 ? (d.bits + EQ_PART - 1) / EQ_PART : 1;
    for (int i = threadIdx.x; i < parts << EQ_PART; i += BLK) {
        const int p = i >> EQ_PART, j = i & ((1 << EQ_PART) - 1), nb = d.bits - EQ_PART * p;
        if (nb < EQ_PART && j >= (1 << nb)) continue;
        E2 f[EQ_PART];
#pragma unroll
        for (int b = 0; b < EQ_PART; b++) {
            f[b] = E2{1, 0};
            if (b < nb) {
                const int c = 2 * (d.first + EQ_PART * p + b);
                const E2 r{set.pt[c], set.pt[c + 1]};
                f[b] = (j >> b) & 1 ? r : F::sub(f[b], r);
            }
        }
        part[p][j] = F::mul(F::mul(F::mul(f[0], f[1]), F::mul(f[2], f[3])), F::mul(F::mul(f[4], f[5]), f[6]));
    }
    __syncthreads();
    uint64_t* out = tabs + d.off;
    for (size_t j = first + threadIdx.x; j < n; j += (size_t)gridDim.y * BLK) {
        E2 x = part[0][j & ((1 << EQ_PART) - 1)];
        for (int p = 1; p < parts; p++) x = F::mul(x, part[p][(j >> (EQ_PART * p)) & ((1 << EQ_PART) - 1)]);
        const uint64_t c0 = F::canon(x.c0), c1 = F::canon(x.c1);
        store2(out + 4 * j, c0, c1);
        store2(out + 4 * j + 2, F::canon(F::times_w(c1)), 0);
    }
}
template <class F>
__device__ __forceinline__ typename F::Pre load_weight(const uint64_t* p) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p);
    return typename F::Pre{a.x, a.y, p[2]};
}

// Sums over the blocks of a grid, in a scratch area of grid_words(entries) words a sum that is zero between kernels: word 0
// counts the blocks that are through, from word 8 on there are four words an entry, the sums of the low and high halves
// of the blocks' canonical words (exact for 2^32 blocks). A block adds its entries with atomics that nobody waits for, so
// the one that finishes last reads each sum once, whatever the grid. (With rows of partial sums it read them all: 148
// rows of 256 entries, 600 KB, took it 7 us; in two levels a fence and a ticket more.) Where there are few sums, blocks add to one
// of several copies: 1184 blocks on the same sixteen sums waited 20 us for one another.
constexpr int ACC_FIRST = 8;
__host__ __device__ constexpr int grid_copies(int entries) { return entries >= 128 ? 1 : entries <= 8 ? 16 : 128 / entries; }
__host__ __device__ constexpr size_t grid_words(int entries) { return ACC_FIRST + 4 * (size_t)entries * grid_copies(entries); }
__device__ __forceinline__ void grid_add(uint64_t* acc, int entries, unsigned block, int entry, uint64_t c0, uint64_t c1) {
    const size_t at = (size_t)(block % grid_copies(entries)) * entries + entry;
    unsigned long long* p = reinterpret_cast<unsigned long long*>(acc + ACC_FIRST + 4 * at);
    atomicAdd(p, (unsigned long long)gl::lo32(c0));
    atomicAdd(p + 1, (unsigned long long)gl::hi32(c0));
    if (c1 != 0) {
        atomicAdd(p + 2, (unsigned long long)gl::lo32(c1));
        atomicAdd(p + 3, (unsigned long long)gl::hi32(c1));
    }
}
template <class F>
__device__ __forceinline__ uint64_t grid_value(uint64_t lo, uint64_t hi) {
    const unsigned __int128 x = ((unsigned __int128)hi << 32) + lo;
    return F::canon(F::red(gl::Acc{(uint32_t)x, (uint32_t)(x >> 32), (uint32_t)(x >> 64), (uint32_t)(x >> 96), 0}));
}
// after every thread's grid_add: true in the block that is through last of the `of` that add (uniform over the block)
__device__ __forceinline__ bool grid_last(uint64_t* acc, bool* flag, unsigned of) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *flag = atomicAdd(reinterpret_cast<unsigned*>(acc), 1u) == of - 1;
    __syncthreads();
    if (!*flag) return false;
    __threadfence();
    if (threadIdx.x == 0) *reinterpret_cast<unsigned*>(acc) = 0;
    return true;
}
// the sum of an entry, which is zero afterwards
template <class F>
__device__ __forceinline__ typename F::E2 grid_take(uint64_t* acc, int entries, int entry) {
    ulonglong2 a = make_ulonglong2(0, 0), b = a;
    ulonglong2* p = reinterpret_cast<ulonglong2*>(acc + ACC_FIRST + 4 * (size_t)entry);
#pragma unroll 4
    for (int c = 0; c < grid_copies(entries); c++, p += 2 * entries) {
        const ulonglong2 x = __ldcg(p), y = __ldcg(p + 1);
        p[0] = p[1] = make_ulonglong2(0, 0);
        a.x += x.x; a.y += x.y; b.x += y.x; b.y += y.y;
    }
    return typename F::E2{grid_value<F>(a.x, a.y), grid_value<F>(b.x, b.y)};
}

// Sums the threads' V values by t mod 2^bits over the block and then over the gridDim.x blocks of blockIdx.y; true in
// the block that finishes last, with the sums (canonical) in sm[0 .. V 2^bits), value j of t at j 2^bits + t.
// acc: grid_words(V 2^bits) words of this blockIdx.y.
template <class F, int V>
__device__ __forceinline__ bool grid_sum(typename F::E2 (&v)[V], int bits, typename F::E2* sm, uint64_t* acc) {
    using E2 = typename F::E2;
    __shared__ bool last;
    const int t = threadIdx.x, n = 1 << bits;
    E2 x[V];
#pragma unroll
    for (int j = 0; j < V; j++) {
        __syncthreads();
        sm[t] = v[j];
        __syncthreads();
        for (int s = BLK / 2; s >= n; s >>= 1) {
            if (t < s) sm[t] = F::add(sm[t], sm[t + s]);
            __syncthreads();
        }
        x[j] = E2{F::canon(sm[t].c0), F::canon(sm[t].c1)};
    }
    if (gridDim.x > 1) {
        if (t < n) {
#pragma unroll
            for (int j = 0; j < V; j++) grid_add(acc, V * n, blockIdx.x, j * n + t, x[j].c0, x[j].c1);
        }
        if (!grid_last(acc, &last, gridDim.x)) return false;
        if (t < n) {
#pragma unroll
            for (int j = 0; j < V; j++) x[j] = grid_take<F>(acc, V * n, j * n + t);
        }
    }
    __syncthreads();
    if (t < n) {
#pragma unroll
        for (int j = 0; j < V; j++) sm[j * n + t] = x[j];
    }
    __syncthreads();
    return true;
}

// ---- the pass -----------------------------------------------------------------------------------------
struct PairArgs {
    int fb;                   // challenges to fold
    const uint64_t *a, *b;    // instance 0's tables: 2^(v + fb) elements, base field words or (c0, c1)
    size_t in_stride;         // words from one instance to the next
    uint64_t* out;            // [instance][a, b][2^v][2] folded tables, or null
    int v;                    // variables left after the fold
    int lo;                   // weighted passes: variables of WL; y's next variables index WH
    int row_shift;            // log2 of the elements between two entries of WH (63: WH is a single 1)
    size_t row_mask;
    const uint64_t *wl, *wh;
    uint64_t* acc;            // [instance][grid_words(4^B)]
    uint64_t* sums;           // pinned: [instance][4^B][2]
};
template <class F>
struct FoldWeights {
    typename F::Pre w[1 << MAX_B];   // eq vector of the challenges to fold, bit k: challenge k
};

// `inputs` terms (two or more, read in pairs) of a folded element from term m0 on, loose: a dot product with the eq vector
template <class F, bool BASE, int UNROLL>
__device__ __forceinline__ typename F::E2 fold_part(const uint64_t* q, int m0, int inputs, const FoldWeights<F>& fw) {
    using E2 = typename F::E2;
    gl::Acc s0 = gl::acc_zero(), s1 = gl::acc_zero();
#pragma unroll UNROLL
    for (int m = 0; m < inputs; m += 2) {
        const typename F::Pre &u = fw.w[m0 + m], &w = fw.w[m0 + m + 1];
        if constexpr (BASE) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(q + m);
            gl::acc_mul(s0, u.c0, v.x);
            gl::acc_mul(s1, u.c1, v.x);
            gl::acc_mul(s0, w.c0, v.y);
            gl::acc_mul(s1, w.c1, v.y);
        } else {
            const E2 v = load2<E2>(q + 2 * m), z = load2<E2>(q + 2 * m + 2);
            gl::acc_mul(s0, u.c0, v.c0);
            gl::acc_mul(s0, u.c1w, v.c1);
            gl::acc_mul(s1, u.c0, v.c1);
            gl::acc_mul(s1, u.c1, v.c0);
            gl::acc_mul(s0, w.c0, z.c0);
            gl::acc_mul(s0, w.c1w, z.c1);
            gl::acc_mul(s1, w.c0, z.c1);
            gl::acc_mul(s1, w.c1, z.c0);
        }
    }
    return E2{F::red(s0), F::red(s1)};
}
// element y of the folded table
template <class F, bool FOLD, bool BASE>
__device__ __forceinline__ typename F::E2 fold_element(const uint64_t* p, size_t y, int fb, const FoldWeights<F>& fw) {
    using E2 = typename F::E2;
    if constexpr (!FOLD) {
        if constexpr (BASE) return E2{p[y], 0};
        else return load2<E2>(p + 2 * y);
    } else {
        const E2 e = fold_part<F, BASE, 2>(p + ((BASE ? y : 2 * y) << fb), 0, 1 << fb, fw);
        return E2{F::canon(e.c0), F::canon(e.c1)};
    }
}
// the sum of 2^s neighbouring threads' parts, canonical
template <class F>
__device__ __forceinline__ typename F::E2 fold_join(typename F::E2 e, int s) {
    for (int off = 1; off < (1 << s); off <<= 1)
        e = F::add(e, typename F::E2{__shfl_xor_sync(0xffffffffu, e.c0, off), __shfl_xor_sync(0xffffffffu, e.c1, off)});
    return typename F::E2{F::canon(e.c0), F::canon(e.c1)};
}

// Small tables as they are, canonical, to page-locked memory: w words of table 2 k + s from (s ? b : a) + stride k. (A copy command
// and a synchronisation took 4 us longer, and as many commands as there were tables.)
template <class F>
__global__ void __launch_bounds__(BLK)
send_tables_kernel(const uint64_t* __restrict__ a, const uint64_t* __restrict__ b, size_t stride, size_t w, uint64_t* out) {
    const uint64_t* p = (blockIdx.y & 1 ? b : a) + stride * (blockIdx.y >> 1);
    for (size_t x = (size_t)blockIdx.x * BLK + threadIdx.x; x < w; x += (size_t)gridDim.x * BLK) out[blockIdx.y * w + x] = F::canon(p[x]);
}

// FOLD: there are challenges to fold (a.fb of them); GB: rounds of the next block (0: fold and store only). BASE: input
// words of the base field.
template <class F, bool FOLD, int GB, bool BASE, bool WEIGHTED>
__global__ void __launch_bounds__(BLK)
pair_pass_kernel(const PairArgs a, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr bool RAW = BASE && !FOLD;                  // b stays a base field element, and a too without weights
    constexpr int E = 1 << (2 * GB);                       // entries of M
    extern __shared__ uint64_t wl_sm[];                    // WEIGHTED: c0[2^lo], c1[2^lo], W c1[2^lo]
    __shared__ E2 sa[BLK], sb[BLK];
    __shared__ uint64_t sbw[BLK];
    const int t = threadIdx.x, k = blockIdx.y;
    const uint64_t *pa = a.a + a.in_stride * k, *pb = a.b + a.in_stride * k;
    uint64_t* oa = a.out ? a.out + ((size_t)4 << a.v) * k : nullptr;
    const size_t n = (size_t)1 << a.v, tiles = (n + BLK - 1) / BLK;
    const size_t per = (tiles + gridDim.x - 1) / gridDim.x, first = per * blockIdx.x;
    const size_t end = first + per < tiles ? first + per : tiles;
    if constexpr (WEIGHTED && GB > 0) {
        const int nl = 1 << a.lo;
        for (int j = t; j < nl; j += BLK) {
            wl_sm[j] = a.wl[4 * j];
            wl_sm[nl + j] = a.wl[4 * j + 1];
            wl_sm[2 * nl + j] = a.wl[4 * j + 2];
        }
        __syncthreads();
    }
    gl::Acc s0 = gl::acc_zero(), s1 = gl::acc_zero();
    E2 sum[1] = {E2{0, 0}};
    const int e = t & (E - 1), ei = (e >> GB) & ((1 << GB) - 1), ej = e & ((1 << GB) - 1), y0 = t >> (2 * GB);
    // without a fold the next tile's elements are loaded before this tile's products
    E2 na{0, 0}, nb{0, 0};
    const auto prefetch = [&](size_t tile) {
        const size_t x = tile * BLK + t;
        if (!FOLD && tile < end && x < n) {
            na = fold_element<F, FOLD, BASE>(pa, x, 0, fw);
            nb = fold_element<F, FOLD, BASE>(pb, x, 0, fw);
        }
    };
    prefetch(first);
    for (size_t tile = first; tile < end; tile++) {
        const size_t x = tile * BLK + t;
        E2 fa = na, fb = nb;
        if constexpr (FOLD) {
            if (x < n) {
                fa = fold_element<F, FOLD, BASE>(pa, x, a.fb, fw);
                fb = fold_element<F, FOLD, BASE>(pb, x, a.fb, fw);
                if (oa != nullptr) {
                    store2(oa + 2 * x, fa.c0, fa.c1);
                    store2(oa + 2 * (n + x), fb.c0, fb.c1);
                }
            }
        } else {
            prefetch(tile + 1);
        }
        if constexpr (GB > 0) {
            if constexpr (WEIGHTED) {
                const int nl = 1 << a.lo, y = (int)((x >> GB) & (nl - 1));
                const typename F::Pre w{wl_sm[y], wl_sm[nl + y], wl_sm[2 * nl + y]};
                gl::Acc c0 = gl::acc_zero(), c1 = gl::acc_zero();
                gl::acc_mul(c0, w.c0, fa.c0);
                gl::acc_mul(c1, w.c1, fa.c0);
                if constexpr (!RAW) {
                    gl::acc_mul(c0, w.c1w, fa.c1);
                    gl::acc_mul(c1, w.c0, fa.c1);
                }
                fa = E2{F::red(c0), F::red(c1)};
            }
            __syncthreads();   // the tile before has been read
            sa[t] = fa;
            sb[t] = fb;
            if constexpr (!RAW) sbw[t] = F::times_w(fb.c1);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < (1 << GB); q++) {
                const int y = (y0 + q * (BLK >> (2 * GB))) << GB;
                const E2 u = sa[y + ei];
                const uint64_t v0 = sb[y + ej].c0;
                gl::acc_mul(s0, u.c0, v0);
                if constexpr (!RAW || WEIGHTED) gl::acc_mul(s1, u.c1, v0);
                if constexpr (!RAW) {
                    gl::acc_mul(s0, u.c1, sbw[y + ej]);
                    gl::acc_mul(s1, u.c0, sb[y + ej].c1);
                }
            }
            if constexpr (WEIGHTED) {
                // the row's WH when the row or the block's share ends
                const size_t row = (tile * BLK) >> a.row_shift;
                if (tile + 1 == end || ((tile + 1) * BLK) >> a.row_shift != row) {
                    sum[0] = F::fma(load_weight<F>(a.wh + 4 * (row & a.row_mask)), E2{F::redw(s0), F::redw(s1)}, sum[0]);
                    s0 = gl::acc_zero();
                    s1 = gl::acc_zero();
                }
            }
        }
    }
    if constexpr (GB > 0) {
        if constexpr (!WEIGHTED) sum[0] = E2{F::redw(s0), F::redw(s1)};
        if (!grid_sum<F, 1>(sum, 2 * GB, sa, a.acc + grid_words(E) * k)) return;
        if (t < E) store2(a.sums + 2 * ((size_t)k * E + t), sa[t].c0, sa[t].c1);
    }
}

// The same for few elements, always with a fold: what takes the time there is one thread's chain (a fold of sixteen inputs is 128 products,
// then sixteen for the sums), on as many SMs as there are tiles of 256 elements. Here 2^s threads share an element of the
// fold and a block takes 128 / 2^s elements of each table, one tile a block. Two tables of 2^13 folded to 2^9 for the host 12.4 -> 6.7 us,
// of 2^16 to 2^13 with the sums of four rounds 12.4 -> 11 us (the atomics over the blocks and the last block are most of it).
template <class F, int GB, bool BASE, bool WEIGHTED>
__global__ void __launch_bounds__(BLK)
pair_small_kernel(const PairArgs a, int s, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr int E = 1 << (2 * GB);
    __shared__ E2 sa[BLK], sb[BLK / 2];
    __shared__ uint64_t sbw[BLK / 2];
    const int t = threadIdx.x, k = blockIdx.y, tile = (BLK / 2) >> s, part = t & ((1 << s) - 1), f = t >> s, x = f & (tile - 1);
    const bool second = f >= tile;   // of the second table
    const size_t n = (size_t)1 << a.v, first = (size_t)blockIdx.x * tile, y = first + x;
    E2 e{0, 0};
    if (y < n) {
        const int inputs = 1 << (a.fb - s), m0 = part * inputs;   // at least two
        e = fold_part<F, BASE, 4>((second ? a.b : a.a) + a.in_stride * k + (((BASE ? y : 2 * y) << a.fb) + (BASE ? m0 : 2 * m0)), m0, inputs, fw);
    }
    e = fold_join<F>(e, s);
    if (part == 0) {
        if (y < n && a.out != nullptr) store2(a.out + ((size_t)4 << a.v) * k + 2 * ((second ? n : 0) + y), e.c0, e.c1);
        if constexpr (GB > 0) {
            if (WEIGHTED && !second && y < n) e = F::fma(load_weight<F>(a.wl + 4 * ((y >> GB) & (((size_t)1 << a.lo) - 1))), e, E2{0, 0});
            if (second) {
                sb[x] = e;
                sbw[x] = F::times_w(e.c1);
            } else {
                sa[x] = e;
            }
        }
    }
    if constexpr (GB > 0) {
        __syncthreads();
        const int entry = t & (E - 1), ei = (entry >> GB) & ((1 << GB) - 1), ej = entry & ((1 << GB) - 1);
        gl::Acc p0 = gl::acc_zero(), p1 = gl::acc_zero();
        for (int b = (t >> (2 * GB)) << GB; b < tile; b += BLK >> GB) {
            const E2 u = sa[b + ei], v = sb[b + ej];
            gl::acc_mul(p0, u.c0, v.c0);
            gl::acc_mul(p0, u.c1, sbw[b + ej]);
            gl::acc_mul(p1, u.c0, v.c1);
            gl::acc_mul(p1, u.c1, v.c0);
        }
        E2 sum[1] = {E2{F::redw(p0), F::redw(p1)}};
        if constexpr (WEIGHTED) {   // a tile lies in one row
            const size_t row = first >> a.row_shift;
            sum[0] = F::fma(load_weight<F>(a.wh + 4 * (row & a.row_mask)), sum[0], E2{0, 0});
        }
        if (!grid_sum<F, 1>(sum, 2 * GB, sa, a.acc + grid_words(E) * k)) return;
        if (t < E) store2(a.sums + 2 * ((size_t)k * E + t), sa[t].c0, sa[t].c1);
    }
}

}  // namespace pr
}  // namespace mb
