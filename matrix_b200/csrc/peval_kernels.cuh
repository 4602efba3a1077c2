// Partial evaluation of a multilinear table: fix its m low variables at r[0..m),
// out[j] = sum_b in[j 2^m + b] eq(r, b), by repeated folding
// T'[y] = T[2y] + r_i (T[2y+1] - T[2y])
// (reference: cuda/partial_eval.cuh:31-219, almost twin
// cuda_almost_goldilocks/almost_partial_eval.cuh:22-180, one launch and one full
// pass per variable). Here m variables take ceil(m / 4) passes and the traffic is
// about N (1 + 2^-4) instead of about 3 N.
//  * The first pass over a base-field table (the large one) is an inner product with the eq vector of the variables it
//    binds, as exact 160-bit sums (two multiply-accumulate chains per element instead of a reduced fold per level):
//    six or more variables by warps that stream whole rows (dot_rows_kernel), of tables of 2^22 elements and more on the
//    tensor cores (peval_mma_kernels.cuh), fewer with the 2^K weights in shared
//    memory (dot_levels_kernel: a block stages 4096 consecutive elements with coalesced 16-byte loads; each thread
//    then reads its run of 2^K from a padded layout without bank conflicts).
//  * Other passes (extension tables, what the first left) fold a run of 2^K
//    consecutive elements through K variables in registers.
#pragma once
#include "peval_mma_kernels.cuh"
#include "sumcheck_kernels.cuh"

namespace mb {
namespace pe {

constexpr int K_MAX = 4;

// Folds variables [lvl, lvl + K): reads 2^K elements of FIn per output, the
// first level lifts FIn to FOut through FoldOp, the others stay in FOut.
// r holds FOut elements.
template <class FIn, class FOut, int K>
__global__ void __launch_bounds__(256)
fold_levels_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, const uint64_t* __restrict__ r, int lvl,
                   size_t n_out) {
    using TI = typename FIn::T;
    using TO = typename FOut::T;
    TO rr[K];
#pragma unroll
    for (int k = 0; k < K; k++) rr[k] = FOut::load(r, lvl + k);
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_out; j += step) {
        TO v[1 << (K - 1)];
#pragma unroll
        for (int p = 0; p < (1 << (K - 1)); p++) {
            TI a, b;
            FIn::load2(in, (j << K) + 2 * p, a, b);
            v[p] = sc::FoldOp<FIn, FOut>::apply(a, b, rr[0]);
        }
#pragma unroll
        for (int k = 1; k < K; k++) {
#pragma unroll
            for (int p = 0; p < (1 << (K - 1 - k)); p++)
                v[p] = sc::FoldOp<FOut, FOut>::apply(v[2 * p], v[2 * p + 1], rr[k]);
        }
        FOut::store(out, j, v[0]);
    }
}

// First pass over a base-field table: K variables at once as an inner product with
// eq weights. One tile = 256 outputs = 256 * 2^K inputs; n_out is a multiple of 256.
template <class FIn, class FOut, int K>
__global__ void __launch_bounds__(256, 4)
dot_levels_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, const uint64_t* __restrict__ r, int lvl,
                  size_t n_out) {
    using TO = typename FOut::T;
    constexpr int R = 1 << K;           // inputs per output
    constexpr int ROW = R + 1;          // padded run in shared memory
    __shared__ uint64_t tile[256 * ROW];
    __shared__ uint64_t wsm[2 * R];     // the weights stay in shared memory: registers are what bounds residency here
    if (threadIdx.x == 0) {
        // w_b = prod_k (b_k ? r_k : 1 - r_k), bit k of b with r[lvl + k]
        TO w[R];
        w[0] = TO{1, 0};
#pragma unroll
        for (int k = 0; k < K; k++) {
            const TO rk = FOut::load(r, lvl + k);
#pragma unroll
            for (int b = 0; b < (1 << k); b++) {
                TO hi = FOut::mul(w[b], rk);
                w[b + (1 << k)] = hi;
                w[b] = FOut::sub(w[b], hi);
            }
        }
#pragma unroll
        for (int b = 0; b < R; b++) FOut::to_words(w[b], wsm + 2 * b);
    }
    __syncthreads();
    const size_t tiles = n_out >> 8;
    for (size_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t* src = in + t * (256 * R);
#pragma unroll
        for (int i = 0; i < R / 2; i++) {
            const int e = 2 * (i * 256 + (int)threadIdx.x);   // element index inside the tile, even
            ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src + e);
            const int row = e >> K, col = e & (R - 1);
            tile[row * ROW + col] = v.x;
            tile[row * ROW + col + 1] = v.y;
        }
        __syncthreads();
        gl::Acc s0 = gl::acc_zero(), s1 = gl::acc_zero();
#pragma unroll
        for (int b = 0; b < R; b++) {
            const uint64_t v = tile[threadIdx.x * ROW + b];
            gl::acc_mul(s0, v, wsm[2 * b]);
            gl::acc_mul(s1, v, wsm[2 * b + 1]);
        }
        FOut::store(out, t * 256 + threadIdx.x, TO{FOut::reduce_acc(s0), FOut::reduce_acc(s1)});
        __syncthreads();
    }
}

// First pass over a base-field table: m >= 6 variables at once. Element b of a row weighs WL[b mod 64] WH[b / 64]: a lane
// keeps elements 2 lane, 2 lane + 1 of every 64, sums them times WH (the same for the whole warp) and applies its two
// entries of WL once at the end, so an element costs two multiply-accumulates whatever m is, and nothing between the
// row and its output goes through memory. 2^parts_log warps of a block share a row. Bound by those products (28 us for
// 2^24 elements) and by the latency of the loads (2^24 elements, m = 12: 55 us at the profiler's clock, where passes of
// four variables took 43 + 11 + 8 and two more launches).
template <class FIn, class FOut>
__global__ void __launch_bounds__(256)
dot_rows_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, const uint64_t* __restrict__ r, int lvl, int m,
                int parts_log, size_t n_out) {
    using TO = typename FOut::T;
    using Sum = sc::NarrowLazy<FIn>;
    extern __shared__ uint64_t wh[];   // [2^(m - 6)][2]
    __shared__ uint64_t part_sm[8][2];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, hi_n = 1 << (m - 6), parts = 1 << parts_log;
    if (t == 0) FOut::to_words(TO{1, 0}, wh);
    __syncthreads();
    for (int k = 0; k < m - 6; k++) {
        const TO rk = FOut::load(r, lvl + 6 + k);
        for (int j = t; j < (1 << k); j += 256) {
            const TO w = FOut::from_words(wh + 2 * j), hi = FOut::mul(w, rk);
            FOut::to_words(FOut::sub(w, hi), wh + 2 * j);
            FOut::to_words(hi, wh + 2 * (j + (1 << k)));
        }
        __syncthreads();
    }
    TO wl0{1, 0};
#pragma unroll
    for (int k = 1; k < 6; k++) {
        const TO rk = FOut::load(r, lvl + k), hi = FOut::mul(wl0, rk);
        wl0 = (lane >> (k - 1)) & 1 ? hi : FOut::sub(wl0, hi);
    }
    const TO wl1 = FOut::mul(wl0, FOut::load(r, lvl));
    wl0 = FOut::sub(wl0, wl1);
    const int rows = 8 >> parts_log, part = warp & (parts - 1);
    for (size_t row0 = (size_t)blockIdx.x * rows; row0 < n_out; row0 += (size_t)gridDim.x * rows) {
        const size_t row = row0 + (warp >> parts_log);   // rows divides n_out
        const uint64_t* src = in + (row << m) + 2 * lane;
        typename Sum::A e0 = Sum::zero(), e1 = Sum::zero(), o0 = Sum::zero(), o1 = Sum::zero();
        // the next four loads are in flight while four are used
        const int count = hi_n >> parts_log;
        const auto index = [&](int k) { return part + ((k & (count - 1)) << parts_log); };   // wraps where there are fewer than four
        ulonglong2 next[4];
#pragma unroll
        for (int u = 0; u < 4; u++) next[u] = *reinterpret_cast<const ulonglong2*>(src + 64 * (size_t)index(u));
        for (int k = 0; k < count; k += 4) {
            ulonglong2 x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = next[u];
            if (k + 4 < count) {
#pragma unroll
                for (int u = 0; u < 4; u++) next[u] = *reinterpret_cast<const ulonglong2*>(src + 64 * (size_t)index(k + 4 + u));
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (k + u >= count) break;
                const int i = index(k + u);
                const uint64_t w0 = wh[2 * i], w1 = wh[2 * i + 1];
                Sum::mul(e0, x[u].x, w0);
                Sum::mul(e1, x[u].x, w1);
                Sum::mul(o0, x[u].y, w0);
                Sum::mul(o1, x[u].y, w1);
            }
        }
        TO v = FOut::add(FOut::mul(TO{Sum::reduce(e0), Sum::reduce(e1)}, wl0), FOut::mul(TO{Sum::reduce(o0), Sum::reduce(o1)}, wl1));
        uint64_t w[2];
        FOut::to_words(v, w);
        const typename FOut::WordAdd wadd;
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            w[0] = wadd(w[0], __shfl_xor_sync(0xffffffffu, w[0], off));
            w[1] = wadd(w[1], __shfl_xor_sync(0xffffffffu, w[1], off));
        }
        if (parts_log == 0) {
            if (lane == 0) FOut::store(out, row, FOut::from_words(w));
            continue;
        }
        if (lane == 0) {
            part_sm[warp][0] = w[0];
            part_sm[warp][1] = w[1];
        }
        __syncthreads();
        if (lane == 0 && part == 0) {
            for (int q = 1; q < parts; q++) {
                w[0] = wadd(w[0], part_sm[warp + q][0]);
                w[1] = wadd(w[1], part_sm[warp + q][1]);
            }
            FOut::store(out, row, FOut::from_words(w));
        }
        __syncthreads();
    }
}
// Variables the first pass binds by rows: all of them unless that leaves fewer than 2^9 rows of a table for which more warps
// are wanted (eight of them share a row at most); at most 14, so that a block's WH stays a few KB. 0: not by rows. A row costs
// the chip about 0.6 ns at its end (five shuffles of two words, two products) whatever its length, so many short rows are
// left to dot_levels_kernel and the passes behind it. Measured, Goldilocks, us by passes of four / by rows: 2^24 elements, m = 6
// (2^18 rows) 65 / 222, m = 9 70 / 78, m = 10 (2^14 rows) 70 / 70, m = 11 72 / 65; 2^21, m = 7 30 / 41, m = 9 (2^12 rows)
// 35 / 30; 2^19, m = 7 (2^12 rows) 27 / 26 (almost-Goldilocks 27 / 29), m = 8 28 / 27: rows of 2^10 elements and more, at most
// 2^12 rows of 2^8 or 2^9, at most 2^11 shorter ones.
inline int dot_rows_vars(int log_n, int m) {
    int k = log_n - 9 > 9 ? log_n - 9 : 9;
    if (k > 14) k = 14;
    if (m < k) k = m;
    return k >= 10 || log_n - k <= (k >= 8 ? 12 : 11) ? k : 0;
}
template <class FIn, class FOut>
inline void launch_dot_rows(const uint64_t* in, uint64_t* out, const uint64_t* r, int lvl, int k, size_t n_out, cudaStream_t st) {
    // eight warps an SM sub-core until the rows alone give them, as long as a warp keeps an iteration
    int parts_log = 0;
    while (parts_log < 3 && (n_out << parts_log) < 4096 && parts_log < k - 6) parts_log++;
    const size_t blocks = (n_out << parts_log) / 8;   // a table of 2^9 elements or more has at least one block's worth
    const size_t cap = (size_t)sm_count() * 8;
    MB_KERNEL_ON("partial_eval_rows", st);
    dot_rows_kernel<FIn, FOut><<<(unsigned)(blocks < cap ? blocks : cap), 256, sizeof(uint64_t) * ((size_t)2 << (k - 6)), st>>>(
        in, out, r, lvl, k, parts_log, n_out);
}

template <class FIn, class FOut>
inline void launch_dot(const uint64_t* in, uint64_t* out, const uint64_t* r, int lvl, int k, size_t n_out, cudaStream_t st) {
    int grid = grid_for(n_out, 256, 4);
    MB_KERNEL_ON("partial_eval_dot", st);
    switch (k) {
        case 1: dot_levels_kernel<FIn, FOut, 1><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        case 2: dot_levels_kernel<FIn, FOut, 2><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        case 3: dot_levels_kernel<FIn, FOut, 3><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        default: dot_levels_kernel<FIn, FOut, 4><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
    }
}

template <class FIn, class FOut>
inline void launch_levels(const uint64_t* in, uint64_t* out, const uint64_t* r, int lvl, int k, size_t n_out,
                          cudaStream_t st) {
    int grid = grid_for(n_out, 256, 8);
    MB_KERNEL_ON("partial_eval_levels", st);
    switch (k) {
        case 1: fold_levels_kernel<FIn, FOut, 1><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        case 2: fold_levels_kernel<FIn, FOut, 2><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        case 3: fold_levels_kernel<FIn, FOut, 3><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
        default: fold_levels_kernel<FIn, FOut, 4><<<grid, 256, 0, st>>>(in, out, r, lvl, n_out); break;
    }
}

struct Plan {
    int first_vars = 0;   // bound by the first pass on the tensor cores or by rows, 0: K_MAX a pass from the start
    bool mma = false;
    int passes = 0;
};
template <class FIn, class FOut>
inline Plan plan(const uint64_t* d_in, int log_n, int m) {
    Plan p;
    // dot_rows_kernel reads pairs of elements, and eight warps of 64 elements or more make a block
    if constexpr (FIn::NW == 1 && FOut::NW == 2)
        if (m >= 6 && log_n >= 9 && (reinterpret_cast<uintptr_t>(d_in) & 15) == 0) {
            p.first_vars = dot_mma_vars(log_n, m);
            p.mma = p.first_vars > 0;
            if (!p.mma) p.first_vars = dot_rows_vars(log_n, m);
        }
    p.passes = p.first_vars ? 1 + (m - p.first_vars + K_MAX - 1) / K_MAX : (m + K_MAX - 1) / K_MAX;
    return p;
}

// d_in: 2^log_n elements of FIn; result: 2^(log_n - m) elements of FOut in
// d_out. d_tmp: scratch of at least 2^(log_n - min(m, K_MAX)) FOut elements
// (unused when m <= K_MAX). d_in is not modified unless it aliases d_out/d_tmp. d_last (may be null): the result goes there, and
// d_out is scratch of three passes and more, d_tmp of two and more (null otherwise).
template <class FIn, class FOut>
inline int partial_eval(const uint64_t* d_in, uint64_t* d_out, uint64_t* d_tmp, const uint64_t* d_r, int log_n, int m,
                        cudaStream_t st, uint64_t* d_last = nullptr) {
    if (log_n < 0 || log_n > 40 || m < 0 || m > log_n || !d_in || (!d_out && !d_last) || (m > 0 && !d_r)) return MB_ERR_ARG;
    if (m == 0) return MB_OK;
    const Plan how = plan<FIn, FOut>(d_in, log_n, m);
    const int first_vars = how.first_vars, passes = how.passes;
    const bool mma = how.mma;
    if ((passes > 1 && !d_tmp) || (passes > 2 && !d_out)) return MB_ERR_ARG;
    // ping-pong so that the last pass lands in d_out
    uint64_t* bufs[2] = {d_out, d_tmp};
    int which = (passes % 2 == 1) ? 0 : 1;
    const uint64_t* src = d_in;
    int lvl = 0, left = m, cur_log = log_n;
    bool first = true;
    while (left > 0) {
        int k = first && first_vars ? first_vars : left < K_MAX ? left : K_MAX;
        size_t n_out = (size_t)1 << (cur_log - k);
        uint64_t* dst = left == k && d_last ? d_last : bufs[which];
        bool done = false;
        if constexpr (FIn::NW == 1 && FOut::NW == 2) {
            if (first && mma) {
                int rc = launch_dot_mma<FOut>(src, dst, d_r, k, n_out, st);
                if (rc != MB_OK) return rc;
                done = true;
            } else if (first && first_vars) {
                launch_dot_rows<FIn, FOut>(src, dst, d_r, lvl, k, n_out, st);
                done = true;
            } else if (first && n_out >= 256) {
                launch_dot<FIn, FOut>(src, dst, d_r, lvl, k, n_out, st);
                done = true;
            }
        }
        if (done) {
        } else if (first) {
            launch_levels<FIn, FOut>(src, dst, d_r, lvl, k, n_out, st);
        } else {
            launch_levels<FOut, FOut>(src, dst, d_r, lvl, k, n_out, st);
        }
        first = false;
        src = dst;
        which ^= 1;
        lvl += k;
        left -= k;
        cur_log -= k;
    }
    return finish_async();
}

}  // namespace pe
}  // namespace mb
