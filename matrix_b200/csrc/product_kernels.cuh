// Several rounds of a sumcheck over a product of one table, or of three or four small ones, per pass.
//
// For sum_x prod_k t_k(x) the next B rounds need nothing of the tables but the 2^(D B) sums
//     T[i_1 .. i_D] = sum_y prod_k t_k(i_k + 2^B y):
// folding and evaluating the round polynomials only combine entries, so the host runs the B rounds on T. A round of
// its own costs a launch, a synchronisation and two reductions whatever its size (about 20 us); T takes 2^((D-1) B)
// products per element instead of the few of a round polynomial, so it is for tables that leave the chip idle: at 2^14
// elements of three tables 2^20 products, 5 us, replace three rounds. Three tables of 2^15 elements and more go to the tensor cores
// (product_mma_kernels.cuh), four of 2^14 and more take a round per pass (sumcheck_kernels.cuh).
//
// One table: the sums by x mod 2^B are a thread's own, its elements lie a multiple of 256 apart.
#pragma once
#include "pair_kernels.cuh"
#include "tcgen05.cuh"

namespace mb {
namespace pr {

struct ProductArgs {
    int fb;               // challenges to fold
    const uint64_t* in;   // D tables of 2^(v + fb) elements, base field words or (c0, c1)
    size_t stride;        // words from one table to the next
    uint64_t* out;        // [D][2^v][2] folded tables, or null
    int v;                // variables left after the fold
    uint64_t* acc;        // grid_words(2^(D B))
    uint64_t* sums;       // pinned: [2^(D B)][2]
};

// One table of 2^6 elements or more. GB = 0: fold and store only.
template <class F, int GB, bool FOLD, bool BASE>
__global__ void __launch_bounds__(BLK)
product_pass_kernel(const ProductArgs a, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    __shared__ E2 sm[BLK];
    const int t = threadIdx.x;
    const size_t n = (size_t)1 << a.v;
    E2 sum[1] = {E2{0, 0}};
#pragma unroll 4
    for (size_t x = (size_t)blockIdx.x * BLK + t; x < n; x += (size_t)gridDim.x * BLK) {
        const E2 f = fold_element<F, FOLD, BASE>(a.in, x, a.fb, fw);
        if (a.out != nullptr) store2(a.out + 2 * x, f.c0, f.c1);
        if constexpr (GB > 0) sum[0] = F::add(sum[0], f);
    }
    if constexpr (GB > 0)
        if (grid_sum<F, 1>(sum, GB, sm, a.acc) && t < (1 << GB)) store2(a.sums + 2 * t, sm[t].c0, sm[t].c1);
}

// Three or four tables. A block takes one tile of PT folded elements of each, 2^s threads to an element's fold. The products of the first
// D - 1 tables are formed once, in shared memory; thread t then owns entry t mod 2^(D B) (two entries that differ in the last index
// where there are more entries than threads) and every 2^(8 - D B)-th y. What is bound here is a thread's chain and then the sums over the
// blocks: the eight blocks of a cluster add theirs through shared memory first, an eighth of the entries each, so that the atomics of
// a pass are those of its clusters. (Every thread with its own products of the first two, tiles of 64, half as many blocks as SMs so that their atomics
// did not take longer than the products: three extension tables of 2^14, fold and three rounds 28.4 -> 15.6 us, of 2^11 13.9 -> 10.8,
// the last fold 8.2 -> 7.2; a proof over tables of 2^14 136 -> 113, over four of 2^13 160 -> 123.)
// n is a multiple of PT, and of 8 PT where there are sums.
constexpr int PRODUCT_CLUSTER = 8;
template <class F, int D, int GB, bool FOLD, bool BASE, int PT>
__global__ void __launch_bounds__(BLK) __cluster_dims__(GB > 0 ? PRODUCT_CLUSTER : 1, 1, 1)
product_tile_kernel(const ProductArgs a, int s, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr int E = 1 << (D * GB), PER = E > BLK ? E / BLK : 1, BITS = E > BLK ? 8 : D * GB;
    constexpr int YS = PT >> GB, PAIRS = 1 << (GB * (D - 1)), MASK = (1 << GB) - 1, CL = PRODUCT_CLUSTER;
    static_assert(PER <= 2 && D * PT <= BLK && (GB == 0 || E >= CL), "a thread owns at most two entries");
    __shared__ E2 sf[D][PT];
    __shared__ __align__(16) E2 work[YS * PAIRS > PER * BLK ? YS * PAIRS : PER * BLK];   // the products, then the block's sums
    __shared__ uint64_t sw[PT];   // W times the last table's second component
    __shared__ bool last;
    const int t = threadIdx.x;
    const size_t n = (size_t)1 << a.v;
    {
        const int part = t & ((1 << s) - 1), k = (t >> s) / PT, x = (t >> s) % PT;
        const size_t g = (size_t)blockIdx.x * PT + x;
        E2 e{0, 0};
        if (k < D) {
            const uint64_t* q = a.in + a.stride * k;
            if constexpr (FOLD) {
                const int inputs = 1 << (a.fb - s), m0 = part * inputs;   // at least two
                e = fold_part<F, BASE, 2>(q + (((BASE ? g : 2 * g) << a.fb) + (BASE ? m0 : 2 * m0)), m0, inputs, fw);
            } else {
                e = fold_element<F, false, BASE>(q, g, 0, fw);
            }
        }
        if constexpr (FOLD) e = fold_join<F>(e, s);
        if (k < D && part == 0) {
            if (a.out != nullptr) store2(a.out + 2 * (n * k + g), e.c0, e.c1);
            sf[k][x] = e;
            if (k == D - 1) sw[x] = F::times_w(e.c1);
        }
    }
    if constexpr (GB > 0) {
        __syncthreads();
        for (int u = t; u < YS * PAIRS; u += BLK) {
            const int b = (u / PAIRS) << GB, i = u % PAIRS;
            E2 q = sf[0][b + (i >> (GB * (D - 2)))];
#pragma unroll
            for (int k = 1; k < D - 1; k++) q = F::mul(q, sf[k][b + ((i >> (GB * (D - 2 - k))) & MASK)]);
            work[u] = q;
        }
        __syncthreads();
        const int e0 = (t & ((1 << BITS) - 1)) * PER;
        gl::Acc s0[PER], s1[PER];
#pragma unroll
        for (int p = 0; p < PER; p++) s0[p] = s1[p] = gl::acc_zero();
        for (int y = t >> BITS; y < YS; y += BLK >> BITS) {
            const E2 q = work[y * PAIRS + (e0 >> GB)];
            const int b = (y << GB) + (e0 & MASK);
#pragma unroll
            for (int p = 0; p < PER; p++) {
                const E2 h = sf[D - 1][b + p];
                gl::acc_mul(s0[p], q.c0, h.c0);
                gl::acc_mul(s0[p], q.c1, sw[b + p]);
                gl::acc_mul(s1[p], q.c0, h.c1);
                gl::acc_mul(s1[p], q.c1, h.c0);
            }
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; p++) work[t * PER + p] = E2{F::red(s0[p]), F::red(s1[p])};   // at most 2^7 products
        for (int h = BLK / 2; h >= E; h >>= 1) {
            __syncthreads();
            if (t < h) work[t] = F::add(work[t], work[t + h]);
        }
        tc::cluster_sync();
        for (int u0 = 0; u0 < E; u0 += BLK) {   // eight threads an entry, one a block
            const int u = u0 + t, from = u % CL, entry = (int)(blockIdx.x % CL) * (E / CL) + u / CL;
            E2 e{0, 0};
            if (u < E) {
                uint32_t at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(tc::smem_u32(&work[entry])), "r"(from));
                asm volatile("ld.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(e.c0), "=l"(e.c1) : "r"(at) : "memory");
            }
            e = fold_join<F>(e, 3);
            if (u < E && from == 0) grid_add(a.acc, E, blockIdx.x / CL, entry, e.c0, e.c1);
        }
        tc::cluster_sync();   // the others have read this block's
        if (!grid_last(a.acc, &last, gridDim.x)) return;
        for (int e = t; e < E; e += BLK) {
            const E2 x = grid_take<F>(a.acc, E, e);
            store2(a.sums + 2 * e, x.c0, x.c1);
        }
    }
}

}  // namespace pr
}  // namespace mb
