// Several rounds of a sumcheck over a product of one table, or of three or four small ones, per pass.
//
// For sum_x prod_k t_k(x) the next B rounds need nothing of the tables but the 2^(D B) sums
//     T[i_1 .. i_D] = sum_y prod_k t_k(i_k + 2^B y):
// folding and evaluating the round polynomials only combine entries, so the host runs the B rounds on T. A round of
// its own costs a launch, a synchronisation and two reductions whatever its size (about 20 us); T takes 2^((D-1) B)
// products per element instead of the few of a round polynomial, so it is for tables that leave the chip idle: at 2^14
// elements of three tables 2^20 products, 8 us, replace three rounds. Three tables of 2^15 elements and more go to the tensor cores
// (product_mma_kernels.cuh), four of 2^14 and more take a round per pass (sumcheck_kernels.cuh).
//
// One table: the sums by x mod 2^B are a thread's own, its elements lie a multiple of 256 apart. Otherwise a block takes
// tiles of 64 folded elements per table in shared memory; thread t owns entry t mod 2^(D B) (two
// entries that differ in the last index where there are more entries than threads) and every 2^(8 - D B)-th y.
#pragma once
#include "pair_kernels.cuh"

namespace mb {
namespace pr {

constexpr int PTILE = 64;

struct ProductArgs {
    int fb;               // challenges to fold
    const uint64_t* in;   // D tables of 2^(v + fb) elements, base field words or (c0, c1)
    size_t stride;        // words from one table to the next
    uint64_t* out;        // [D][2^v][2] folded tables, or null
    int v;                // variables left after the fold, at least 6
    uint64_t* acc;        // grid_words(2^(D B))
    uint64_t* sums;       // pinned: [2^(D B)][2]
};

// GB = 0: fold and store only.
template <class F, int D, int GB, bool FOLD, bool BASE>
__global__ void __launch_bounds__(BLK)
product_pass_kernel(const ProductArgs a, const __grid_constant__ FoldWeights<F> fw) {
    using E2 = typename F::E2;
    constexpr int E = 1 << (D * GB), PER = E > BLK ? E / BLK : 1, BITS = E > BLK ? 8 : D * GB;
    static_assert(PER <= 2, "a thread owns at most two entries");
    __shared__ E2 sm[PER * BLK];
    const int t = threadIdx.x;
    const size_t n = (size_t)1 << a.v;
    if constexpr (D == 1) {
        E2 sum[1] = {E2{0, 0}};
#pragma unroll 4
        for (size_t x = (size_t)blockIdx.x * BLK + t; x < n; x += (size_t)gridDim.x * BLK) {
            const E2 f = fold_element<F, FOLD, BASE>(a.in, x, a.fb, fw);
            if (a.out != nullptr) store2(a.out + 2 * x, f.c0, f.c1);
            if constexpr (GB > 0) sum[0] = F::add(sum[0], f);
        }
        if constexpr (GB > 0)
            if (grid_sum<F, 1>(sum, GB, sm, a.acc) && t < E) store2(a.sums + 2 * t, sm[t].c0, sm[t].c1);
        return;
    }
    __shared__ E2 s[D][PTILE];
    __shared__ uint64_t sw[PTILE];   // W times the last table's second component
    const size_t tiles = n / PTILE;
    const int e0 = (t & ((1 << BITS) - 1)) * PER, y0 = t >> BITS;
    int idx[D];
#pragma unroll
    for (int k = 0; k < D; k++) idx[k] = (e0 >> (GB * (D - 1 - k))) & ((1 << GB) - 1);
    gl::Acc s0[PER], s1[PER];
#pragma unroll
    for (int p = 0; p < PER; p++) s0[p] = s1[p] = gl::acc_zero();
    for (size_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();   // the tile before has been read
        for (int j = t; j < D * PTILE; j += BLK) {
            const int k = j / PTILE, x = j % PTILE;
            const size_t g = tile * PTILE + x;
            const E2 f = fold_element<F, FOLD, BASE>(a.in + a.stride * k, g, a.fb, fw);
            if (a.out != nullptr) store2(a.out + 2 * (n * k + g), f.c0, f.c1);
            s[k][x] = f;
            if (k == D - 1) sw[x] = F::times_w(f.c1);
        }
        __syncthreads();
        if constexpr (GB > 0) {
            for (int y = y0; y < (PTILE >> GB); y += BLK >> BITS) {
                const int b = y << GB;
                E2 q = s[0][b + idx[0]];
#pragma unroll
                for (int k = 1; k < D - 1; k++) q = F::mul(q, s[k][b + idx[k]]);
#pragma unroll
                for (int p = 0; p < PER; p++) {
                    const E2 h = s[D - 1][b + idx[D - 1] + p];
                    gl::acc_mul(s0[p], q.c0, h.c0);
                    gl::acc_mul(s0[p], q.c1, sw[b + idx[D - 1] + p]);
                    gl::acc_mul(s1[p], q.c0, h.c1);
                    gl::acc_mul(s1[p], q.c1, h.c0);
                }
            }
        }
    }
    if constexpr (GB > 0) {
        E2 sum[PER];
#pragma unroll
        for (int p = 0; p < PER; p++) sum[p] = E2{F::redw(s0[p]), F::redw(s1[p])};
        if (grid_sum<F, PER>(sum, BITS, sm, a.acc) && t < (1 << BITS)) {
#pragma unroll
            for (int p = 0; p < PER; p++) store2(a.sums + 2 * (size_t)(t * PER + p), sm[(p << BITS) + t].c0, sm[(p << BITS) + t].c1);
        }
    }
}

}  // namespace pr
}  // namespace mb
