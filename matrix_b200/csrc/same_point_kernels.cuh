// Kernels of the same-point sumcheck with the eq polynomials kept factored (almost-Goldilocks, X^2 = 3).
//
// Leaf i proves sum_x eq(r_i, x) f_i(x). Round j binds variable j, the low index bit. With eq a product over the
// variables, B consecutive rounds starting at variable o need nothing of the tables but the 2^B sums
//     G(m) = sum_y eq((r_{o+B}, ..), y) f(m + 2^B y)            (f: the table after o rounds),
// because those rounds only fold and weight the low B variables. So a pass over a table serves B rounds: it folds
// the B challenges of the rounds before (one product per element read, a dot product with their eq vector, reduced
// once), stores the folded table, and adds every folded value times its eq weight to the next G. The eq tables
// themselves (as large as the witness, in extension elements) are never formed: a weight is WL[t] WH[i] with t a
// thread's fixed low index and i its loop counter, so the sum over i is taken with WH (one value for the whole block)
// and multiplied by WL once at the end.
//
// A packed witness stays packed for six rounds: G over the six variables inside a 64-bit word is a set of selected
// additions (bits_pass), and the first extension table, 1/64 of the witness, comes from eight table look-ups per
// word (fold_pass with SRC 1 or 2).
//
// The B rounds' polynomial over all leaves, sum_i scale_i prod_j eq(r_ij, c_j) G_i(c), has degree two in each variable, so
// 3^B values (at 0, 1 and infinity) hold it: the block that finishes a leaf's G multiplies it out and adds it to the others'
// (leaf_share), and the host runs the rounds on at most 81 elements, whatever the number of leaves.
//
// Arity 22, 42 binary leaves: what the proof reads from DRAM is the 22 MB of bits; the largest table is 44 MB.
// bits_pass is bound by the integer pipe (18 instructions per word and warp), the other passes by launch latency.
#pragma once
#include "agl_traits.cuh"
#include "pair_kernels.cuh"

namespace mb {
namespace sp {

using agl::E2;
using agl::E2Pre;

constexpr int BLK = 256;
constexpr int BITS = 6;        // variables inside a packed word
constexpr int MAX_B = 4;       // rounds per pass over a table

// ---- eq tables -----------------------------------------------------------------------------------
// Table d: eq over variables [first, first + bits) of every leaf's point, entries (c0, c1, 3 c1, 0) at word
// offset `off` of the leaf's area.
struct TableDesc {
    int first, bits;
    size_t off;
};
constexpr int MAX_TABLES = 40;
struct TableSet {
    TableDesc d[MAX_TABLES];
};
__device__ __forceinline__ E2Pre load_weight(const uint64_t* p) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p);
    return E2Pre{a.x, a.y, p[2]};
}
static __global__ void __launch_bounds__(BLK)
eq_tables_kernel(const __grid_constant__ TableSet set, const uint64_t* __restrict__ pts, int arity, uint64_t* __restrict__ tabs,
                 size_t leaf_words) {
    const TableDesc d = set.d[blockIdx.x];
    const uint64_t* r = pts + 2 * (size_t)arity * blockIdx.y;
    uint64_t* out = tabs + leaf_words * blockIdx.y + d.off;
    if (threadIdx.x == 0) agl::e2_store(out, E2{1, 0});
    __syncthreads();
    for (int b = 0; b < d.bits; b++) {
        const E2 rb = agl::e2_load(r + 2 * (d.first + b));
        const size_t half = (size_t)1 << b;
        for (size_t j = threadIdx.x; j < half; j += BLK) {
            const E2 a = agl::e2_load(out + 4 * j), ar = agl::e2_mul_lazy(a, rb);
            agl::e2_store(out + 4 * j, agl::e2_canon(agl::e2_sub(a, ar)));
            agl::e2_store(out + 4 * (j + half), agl::e2_canon(ar));
        }
        __syncthreads();
    }
    for (size_t j = threadIdx.x; j < ((size_t)1 << d.bits); j += BLK)
        agl::e2_store(out + 4 * j + 2, E2{agl::canon(agl::mul_small(out[4 * j + 1], 3)), 0});
}

// ---- sums ------------------------------------------------------------------------------------------
// (s0, s1) += w f as exact sums
__device__ __forceinline__ void weigh(gl::Acc& s0, gl::Acc& s1, const E2Pre& w, E2 f) {
    gl::acc_mul(s0, w.c0, f.c0);
    gl::acc_mul(s0, w.c1w, f.c1);
    gl::acc_mul(s1, w.c0, f.c1);
    gl::acc_mul(s1, w.c1, f.c0);
}

// Adds the threads' values v by t mod 2^bits over the block, then over the leaf's gridDim.x blocks; the block that
// finishes last gets true, with the 2^bits sums in sm[0 .. 2^bits) (canonical). partial: the leaf's area of
// gridDim.x * 2^bits elements; counter: the leaf's, zero before and after. sm: BLK elements.
__device__ __forceinline__ bool leaf_sum(E2 v, int bits, E2* sm, uint64_t* partial, unsigned* counter) {
    __shared__ bool last;
    const int t = threadIdx.x, n = 1 << bits;
    const auto block_sum = [&](E2 x) {
        __syncthreads();
        sm[t] = x;
        __syncthreads();
        for (int s = BLK / 2; s >= n; s >>= 1) {
            if (t < s) sm[t] = agl::e2_add(sm[t], sm[t + s]);
            __syncthreads();
        }
        if (t < n) sm[t] = agl::e2_canon(sm[t]);
        __syncthreads();
    };
    block_sum(v);
    if (gridDim.x == 1) return true;
    if (t < n) {
        agl::e2_store(partial + 2 * ((size_t)blockIdx.x * n + t), sm[t]);
        __threadfence();
    }
    __syncthreads();
    if (t == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    E2 x{0, 0};
    for (unsigned b = t >> bits; b < gridDim.x; b += BLK >> bits) {
        const uint64_t* p = partial + 2 * ((size_t)b * n + (t & (n - 1)));
        x = agl::e2_add(x, E2{__ldcg(p), __ldcg(p + 1)});
    }
    block_sum(x);
    if (t == 0) *counter = 0;
    return true;
}

// ---- the rounds' polynomial over the leaves -----------------------------------------------------------
constexpr int SHARE = 81;      // 3^MAX_B
// Leaf share of the values at {0, 1, inf}^B, variable 0 the lowest digit, from the leaf's 2^B sums g (shared memory), added to the
// other leaves'; the block that adds the last one writes them to u (pinned) and leaves acc zero. r: the leaf's
// coordinates of the B variables; acc: pr::grid_words(3^B).
__device__ __forceinline__ void leaf_share(const E2* g, int B, const uint64_t* r, E2 scale, unsigned leaf, unsigned leaves, uint64_t* acc, uint64_t* u) {
    __shared__ E2 f[3 * MAX_B], buf[2][SHARE];
    __shared__ bool last;
    const int t = threadIdx.x;
    if (t < 3 * B) {   // c^0 .. : 1 - r at 0, r at 1, 2 r - 1 the coefficient of c^2 with g(1) - g(0)
        const E2 x = agl::e2_load(r + 2 * (t / 3)), one{1, 0};
        E2 v = t % 3 == 0 ? agl::e2_sub(one, x) : t % 3 == 1 ? x : agl::e2_sub(agl::e2_add(x, x), one);
        if (t < 3) v = agl::e2_mul_lazy(v, scale);
        f[t] = v;
    }
    __syncthreads();
    int low = 1, high = 1 << (B - 1);
    for (int j = 0; j < B; j++, low *= 3, high /= 2) {
        const E2* in = j == 0 ? g : buf[(j - 1) & 1];
        if (t < 3 * low * high) {
            const int l = t % low, p = (t / low) % 3, h = t / (3 * low);
            const E2 g0 = in[l + low * 2 * h], g1 = in[l + low * (2 * h + 1)];
            buf[j & 1][t] = agl::e2_mul_lazy(f[3 * j + p], p == 0 ? g0 : p == 1 ? g1 : agl::e2_sub(g1, g0));
        }
        __syncthreads();
    }
    if (t < low) {
        const E2 v = agl::e2_canon(buf[(B - 1) & 1][t]);
        pr::grid_add(acc, low, leaf, t, v.c0, v.c1);
    }
    if (!pr::grid_last(acc, &last, leaves)) return;
    if (t < low) agl::e2_store(u + 2 * t, pr::grid_take<pr::AglF>(acc, low, t));
}
// The same for the sums of the first pass, which is queued before alpha is known: leaf i's scale is alpha^i.
static __global__ void __launch_bounds__(BLK)
first_share_kernel(const uint64_t* __restrict__ sums, int B, const uint64_t* __restrict__ pts, int arity, E2 alpha,
                   uint64_t* __restrict__ scale, uint64_t* acc, uint64_t* u) {
    __shared__ E2 g[1 << MAX_B];
    const int leaf = blockIdx.x, t = threadIdx.x;
    if (t < (1 << B)) g[t] = agl::e2_load(sums + 2 * (((size_t)leaf << B) + t));
    E2 s{1, 0}, p = alpha;
    for (int e = leaf; e > 0; e >>= 1) {
        if (e & 1) s = agl::e2_mul_lazy(s, p);
        if (e > 1) p = agl::e2_mul_lazy(p, p);
    }
    if (t == 0) agl::e2_store(scale + 2 * (size_t)leaf, agl::e2_canon(s));
    __syncthreads();
    leaf_share(g, B, pts + 2 * (size_t)arity * leaf, s, leaf, gridDim.x, acc, u);
}

// ---- pass over the packed words ----------------------------------------------------------------------
struct BitsArgs {
    const uint64_t *pos, *neg;      // [leaf][words]
    size_t words;                   // per leaf
    int lo_bits, hi_bits;           // words = 2^(lo_bits + hi_bits)
    int in_bits;                    // variables inside a word (fewer than six only for a single word)
    int first_bits;                 // variables of the G that goes to the host
    const uint64_t* tabs;           // eq tables, leaf_words per leaf
    size_t leaf_words, wl_off, wh_off, low_off;   // over the low, the high word variables; over variables [first_bits, in_bits)
    uint64_t *partial, *g6;         // [leaf][gridDim.x][64][2]; [leaf][64][2] = the sums over all words
    unsigned* counter;
    uint64_t* out;                  // pinned: [leaf][2^first_bits][2]
};
// a += e where the bit is set: 96-bit sums per component
__device__ __forceinline__ void add_if(uint32_t (&a)[6], uint32_t word, uint32_t mask, ulonglong2 e) {
    asm("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\tand.b32 t, %6, %7;\n\tsetp.ne.u32 p, t, 0;\n\t"
        "@p add.cc.u32 %0, %0, %8;\n\t@p addc.cc.u32 %1, %1, %9;\n\t@p addc.u32 %2, %2, 0;\n\t"
        "@p add.cc.u32 %3, %3, %10;\n\t@p addc.cc.u32 %4, %4, %11;\n\t@p addc.u32 %5, %5, 0;\n\t}"
        : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5])
        : "r"(word), "r"(mask), "r"(gl::lo32(e.x)), "r"(gl::hi32(e.x)), "r"(gl::lo32(e.y)), "r"(gl::hi32(e.y)));
}
__device__ __forceinline__ E2 sum96(const uint32_t (&a)[6]) {
    return E2{agl::reduce_limbs(a[0], a[1], a[2], 0), agl::reduce_limbs(a[3], a[4], a[5], 0)};
}
// Warp per high index: its 2^lo_bits words against WL, lane l keeps the sums of bit positions l and l + 32.
template <bool TERNARY>
__global__ void __launch_bounds__(BLK)
bits_pass_kernel(const BitsArgs a) {
    __shared__ ulonglong2 wl[1 << 8];
    __shared__ uint64_t stage[BLK / 32][TERNARY ? 2 : 1][32];
    __shared__ E2 sm[BLK];
    __shared__ E2 acc[BLK / 32][64];
    const int leaf = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_lo = 1 << a.lo_bits;
    const uint64_t* tabs = a.tabs + a.leaf_words * leaf;
    for (int j = threadIdx.x; j < n_lo; j += BLK) wl[j] = *reinterpret_cast<const ulonglong2*>(tabs + a.wl_off + 4 * j);
    __syncthreads();
    const size_t n_hi = (size_t)1 << a.hi_bits;
    const uint64_t keep = a.in_bits == BITS ? ~0ULL : ((1ULL << (1 << a.in_bits)) - 1);
    const uint32_t mask = 1u << lane;
    E2 s0{0, 0}, s1{0, 0};
    for (size_t hi = (size_t)blockIdx.x * (BLK / 32) + warp; hi < n_hi; hi += (size_t)gridDim.x * (BLK / 32)) {
        uint32_t p0[6] = {0, 0, 0, 0, 0, 0}, p1[6] = {0, 0, 0, 0, 0, 0}, q0[6] = {0, 0, 0, 0, 0, 0}, q1[6] = {0, 0, 0, 0, 0, 0};
        const size_t base = a.words * leaf + (hi << a.lo_bits);
        for (int j0 = 0; j0 < n_lo; j0 += 32) {
            __syncwarp();
            if (j0 + lane < n_lo) {
                stage[warp][0][lane] = a.pos[base + j0 + lane] & keep;
                if (TERNARY) stage[warp][1][lane] = a.neg[base + j0 + lane] & keep;
            }
            __syncwarp();
            const int cnt = n_lo - j0 < 32 ? n_lo - j0 : 32;
#pragma unroll 4
            for (int j = 0; j < cnt; j++) {
                const ulonglong2 e = wl[j0 + j];
                const uint64_t w = stage[warp][0][j];
                add_if(p0, gl::lo32(w), mask, e);
                add_if(p1, gl::hi32(w), mask, e);
                if (TERNARY) {
                    const uint64_t m = stage[warp][1][j];
                    add_if(q0, gl::lo32(m), mask, e);
                    add_if(q1, gl::hi32(m), mask, e);
                }
            }
        }
        const E2Pre wh = load_weight(tabs + a.wh_off + 4 * hi);
        E2 x0 = sum96(p0), x1 = sum96(p1);
        if (TERNARY) { x0 = agl::e2_sub(x0, sum96(q0)); x1 = agl::e2_sub(x1, sum96(q1)); }
        s0 = agl::e2_fma_pre(wh, x0, s0);
        s1 = agl::e2_fma_pre(wh, x1, s1);
    }
    acc[warp][lane] = s0;
    acc[warp][lane + 32] = s1;
    __syncthreads();
    const int t = threadIdx.x;   // 4 threads per bit position, two warps' sums each
    const E2 v = agl::e2_add(acc[2 * (t >> 6)][t & 63], acc[2 * (t >> 6) + 1][t & 63]);
    if (!leaf_sum(v, BITS, sm, a.partial + 2 * 64 * (size_t)gridDim.x * leaf, a.counter + leaf)) return;
    if (t < 64) agl::e2_store(a.g6 + 2 * (64 * (size_t)leaf + t), sm[t]);
    if (t < (1 << a.first_bits)) {
        E2 g{0, 0};
        for (int k = 0; k < (1 << (a.in_bits - a.first_bits)); k++)
            g = agl::e2_fma_pre(load_weight(tabs + a.low_off + 4 * k), sm[t + (k << a.first_bits)], g);
        agl::e2_store(a.out + 2 * (((size_t)leaf << a.first_bits) + t), agl::e2_canon(g));
    }
}

// ---- pass over an extension table (or the words, the first time) -----------------------------------------
struct FoldArgs {
    const uint64_t *in, *neg;       // SRC 0: [leaf][2^(v + B)][2]; 1: packed words; 2: masks of +1 (in) and -1 (neg)
    size_t in_stride;               // words per leaf
    uint64_t* table;                // [leaf][2^v][2], or null
    int v;                          // variables left after the fold
    int t_bits;                     // min(v, 8): outputs of one block iteration
    int next;                       // rounds of the next G (next <= t_bits)
    const uint64_t* tabs;
    size_t leaf_words, wl_off, wh_off;   // over variables next .. t_bits and t_bits .. v of the folded table
    uint64_t* partial;              // [leaf][gridDim.x][2^next][2]
    unsigned* counter;
    uint64_t* out;                  // pinned: [leaf][2^next][2], or null
    // SHARE_OUT: the rounds' polynomial; scale_i takes in `bound` variables from first - bound on
    const uint64_t* pts;
    int arity, first, bound;        // first: the variable the stage starts at
    uint64_t *scale, *acc, *u;      // [leaf][2]; pr::grid_words(3^next); pinned: [3^next][2]
    E2 r[MAX_B];                    // their challenges
};
struct FoldWeights {
    E2Pre w[1 << MAX_B];            // eq of the challenges, index bit k: challenge k
};
struct WordWeights {
    E2 w[64];
};
// one byte's worth of selected additions: 256 entries per byte of a word
__device__ __forceinline__ void add_entry(gl::Acc& c0, gl::Acc& c1, ulonglong2 e) {
    gl::acc_add(c0, e.x);
    gl::acc_add(c1, e.y);
}
// SHARE_OUT: the leaf's share of the rounds' polynomial too (the code and its shared memory cost the other form 3 us a pass)
template <int B, int SRC, bool SHARE_OUT, class W>
__global__ void __launch_bounds__(BLK)
fold_pass_kernel(const FoldArgs a, const __grid_constant__ W fw) {
    extern __shared__ ulonglong2 lut[];   // SRC > 0: [8][256]
    __shared__ E2 sm[BLK];
    const int leaf = blockIdx.y, t = threadIdx.x;
    const uint64_t* tabs = a.tabs + a.leaf_words * leaf;
    const uint64_t* in = a.in + a.in_stride * leaf;
    const uint64_t* neg = SRC == 2 ? a.neg + a.in_stride * leaf : nullptr;
    if constexpr (SRC > 0) {
        if (t < 8) lut[256 * t] = make_ulonglong2(0, 0);
        __syncthreads();
        for (int b = 0; b < 8; b++) {
            for (int k = t; k < 8 << b; k += BLK) {
                const int byte = k >> b, low = k & ((1 << b) - 1);
                const ulonglong2 e = lut[256 * byte + low];
                const E2 s = agl::e2_canon(agl::e2_add(E2{e.x, e.y}, fw.w[8 * byte + b]));
                lut[256 * byte + low + (1 << b)] = make_ulonglong2(s.c0, s.c1);
            }
            __syncthreads();
        }
    }
    const size_t n = (size_t)1 << a.v, iters = a.v > a.t_bits ? n >> a.t_bits : 1;
    gl::Acc s0 = gl::acc_zero(), s1 = gl::acc_zero();
    E2 single{0, 0};
    for (size_t i = blockIdx.x; i < iters; i += gridDim.x) {
        const size_t y = (i << a.t_bits) + t;
        if (y >= n) break;           // only when a block has more threads than the table has elements
        E2 f;
        if constexpr (SRC == 0 && B == 0) {
            f = agl::e2_load(in + 2 * y);
        } else if constexpr (SRC == 0) {
            gl::Acc c0 = gl::acc_zero(), c1 = gl::acc_zero();
            const uint64_t* p = in + ((2 * y) << B);
#pragma unroll
            for (int m = 0; m < (1 << B); m++) weigh(c0, c1, fw.w[m], agl::e2_load(p + 2 * m));
            f = agl::e2_canon(E2{agl::acc_reduce(c0), agl::acc_reduce(c1)});
        } else {
            gl::Acc c0 = gl::acc_zero(), c1 = gl::acc_zero();
            const uint64_t w = in[y];
#pragma unroll
            for (int b = 0; b < 8; b++) add_entry(c0, c1, lut[256 * b + ((w >> (8 * b)) & 255)]);
            f = E2{agl::acc_reduce(c0), agl::acc_reduce(c1)};
            if constexpr (SRC == 2) {
                c0 = gl::acc_zero();
                c1 = gl::acc_zero();
                const uint64_t m = neg[y];
#pragma unroll
                for (int b = 0; b < 8; b++) add_entry(c0, c1, lut[256 * b + ((m >> (8 * b)) & 255)]);
                f = agl::e2_sub(f, E2{agl::acc_reduce(c0), agl::acc_reduce(c1)});
            }
            f = agl::e2_canon(f);
        }
        if (a.table != nullptr) agl::e2_store(a.table + 2 * (n * leaf + y), f);
        if (iters == 1) single = f;
        else weigh(s0, s1, load_weight(tabs + a.wh_off + 4 * i), f);
    }
    if (iters > 1) single = E2{agl::acc_reduce_wide(s0), agl::acc_reduce_wide(s1)};
    if (a.next < a.t_bits && t < (1 << a.t_bits))
        single = agl::e2_fma_pre(load_weight(tabs + a.wl_off + 4 * (t >> a.next)), single, E2{0, 0});
    if (!leaf_sum(single, a.next, sm, a.partial + ((size_t)(2 * gridDim.x) << a.next) * leaf, a.counter + leaf)) return;
    if (a.out != nullptr && t < (1 << a.next)) agl::e2_store(a.out + 2 * (((size_t)leaf << a.next) + t), sm[t]);
    if constexpr (SHARE_OUT) {
        __shared__ E2 f[MAX_B];
        const uint64_t* pts = a.pts + 2 * ((size_t)a.arity * leaf + a.first);
        if (t < MAX_B) {   // eq(r, R) = 1 - r - R + 2 r R
            E2 v{1, 0};
            if (t < a.bound) {
                const E2 x = agl::e2_load(pts + 2 * (t - a.bound)), xr = agl::e2_mul_lazy(x, a.r[t]);
                v = agl::e2_add(agl::e2_sub(agl::e2_sub(v, x), a.r[t]), agl::e2_add(xr, xr));
            }
            f[t] = v;
        }
        __syncthreads();
        const E2 scale = agl::e2_canon(agl::e2_mul_lazy(agl::e2_mul_lazy(agl::e2_mul_lazy(f[0], f[1]), agl::e2_mul_lazy(f[2], f[3])),
                                                        agl::e2_load(a.scale + 2 * (size_t)leaf)));
        __syncthreads();
        if (t == 0) agl::e2_store(a.scale + 2 * (size_t)leaf, scale);
        leaf_share(sm, a.next, pts, scale, leaf, gridDim.y, a.acc, a.u);
    }
}

}  // namespace sp
}  // namespace mb
