// Multilinear sumcheck kernels, generic over the field (a traits class).
//
// Work per round of the linear sumcheck (reference kernels
// cuda/sumcheck_prover.cuh:37-151,171-292 and the almost-Goldilocks twins
// cuda_almost_goldilocks/almost_sumcheck_prover.cuh:24-218):
//   message  P(c) = sum_y prod_i (a_i + c (b_i - a_i)),  c = 0..D,
//            a_i = T_i[2y], b_i = T_i[2y+1]
//   fold     T_i'[y] = a_i + r (b_i - a_i)
// The reference launches these as two kernels per round, so every table is read
// twice. Here the fold on challenge r_k is fused with the message of round k+1:
// one pass reads four consecutive elements per table, writes the two folded
// ones and accumulates the next message from them, so each round streams the
// tables through HBM once (read S, write S/2).
//
// Tables are poly-major with a fixed stride (the original table length), the
// layout of GpuSumcheckState (goldilocks-cuda-rs/src/sumcheck_prover.rs:20-28).
// Everything written to global memory is canonical.
#pragma once
#include "common.cuh"
#include "gl_field.cuh"

namespace mb {
namespace sc {

constexpr int BLOCK = 256;
constexpr int MAX_D = 8;  // cuda/sumcheck_prover.cuh:18-19

// ---- field traits ---------------------------------------------------------
// WordAdd / WordCanon act on single u64 residues of the base field; block
// reductions use them on the flattened words of an element.
struct GlAdd {
    __device__ __forceinline__ uint64_t operator()(uint64_t a, uint64_t b) const { return gl::add(a, b); }
};
struct GlCanon {
    __host__ __device__ __forceinline__ uint64_t operator()(uint64_t a) const { return gl::canon(a); }
};

struct GlBase {
    using T = uint64_t;
    using WordAdd = GlAdd;
    using WordCanon = GlCanon;
    static constexpr int NW = 1;
    static __device__ __forceinline__ T load(const uint64_t* p, size_t i) { return p[i]; }
    static __device__ __forceinline__ void load2(const uint64_t* p, size_t i, T& a, T& b) {
        ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + i);
        a = v.x; b = v.y;
    }
    static __device__ __forceinline__ void store(uint64_t* p, size_t i, T v) { p[i] = gl::canon(v); }
    static __device__ __forceinline__ void store2(uint64_t* p, size_t i, T a, T b) {
        *reinterpret_cast<ulonglong2*>(p + i) = make_ulonglong2(gl::canon(a), gl::canon(b));
    }
    static __device__ __forceinline__ T add(T a, T b) { return gl::add(a, b); }
    static __device__ __forceinline__ T sub(T a, T b) { return gl::sub(a, b); }
    static __device__ __forceinline__ T mul(T a, T b) { return gl::mul(a, b); }
    static __device__ __forceinline__ T zero() { return 0; }
    static __device__ __forceinline__ void to_words(T v, uint64_t* w) { w[0] = v; }
    static __device__ __forceinline__ T from_words(const uint64_t* w) { return w[0]; }
    // a factor used many times (nothing to prepare in the base field)
    using Pre = uint64_t;
    static __device__ __forceinline__ Pre pre(T x) { return x; }
    static __device__ __forceinline__ T mul_pre(Pre p, T x) { return gl::mul(p, x); }
};

struct GlExt2 {
    using T = gl::E2;
    using WordAdd = GlAdd;
    using WordCanon = GlCanon;
    static constexpr int NW = 2;
    static __device__ __forceinline__ T load(const uint64_t* p, size_t i) { return gl::e2_load(p + 2 * i); }
    static __device__ __forceinline__ void load2(const uint64_t* p, size_t i, T& a, T& b) {
        a = gl::e2_load(p + 2 * i);
        b = gl::e2_load(p + 2 * i + 2);
    }
    static __device__ __forceinline__ void store(uint64_t* p, size_t i, T v) {
        gl::e2_store(p + 2 * i, gl::e2_canon(v));
    }
    static __device__ __forceinline__ void store2(uint64_t* p, size_t i, T a, T b) {
        store(p, i, a);
        store(p, i + 1, b);
    }
    static __device__ __forceinline__ T add(T a, T b) { return gl::e2_add(a, b); }
    static __device__ __forceinline__ T sub(T a, T b) { return gl::e2_sub(a, b); }
    static __device__ __forceinline__ T mul(T a, T b) { return gl::e2_mul_lazy(a, b); }
    static __device__ __forceinline__ T zero() { return gl::E2{0, 0}; }
    static __device__ __forceinline__ void to_words(T v, uint64_t* w) { w[0] = v.c0; w[1] = v.c1; }
    static __device__ __forceinline__ T from_words(const uint64_t* w) { return T{w[0], w[1]}; }
    // a factor used many times, with its c1 times the non-residue prepared: four products, two reductions
    using Pre = gl::E2Pre;
    static __device__ __forceinline__ Pre pre(T x) { return gl::e2_pre(x); }
    static __device__ __forceinline__ T mul_pre(Pre p, T x) { return gl::e2_mul_pre(p, x); }
    // an exact sum of at most 64 products of 64-bit words, reduced to a loose residue
    static __device__ __forceinline__ uint64_t reduce_acc(const gl::Acc& s) { return gl::acc_reduce(s); }
};

// Exact sums of products for a field: A holds sum x_k y_k without any reduction, any number of products. The non-residue is
// multiplied into the second factor first, so an extension element takes two sums. Specialised per field (almost-Goldilocks in
// agl_traits.cuh).
template <class F>
struct NarrowLazy;
struct NarrowSum {
    gl::Acc s0, s1;
};
template <>
struct NarrowLazy<GlBase> {
    using A = gl::Acc;
    static __device__ __forceinline__ A zero() { return gl::acc_zero(); }
    static __device__ __forceinline__ void mul(A& s, uint64_t x, uint64_t y) { gl::acc_mul(s, x, y); }
    static __device__ __forceinline__ uint64_t reduce(const A& s) { return gl::acc_reduce_wide(s); }
};
template <>
struct NarrowLazy<GlExt2> {
    using A = NarrowSum;
    static __device__ __forceinline__ A zero() { return A{gl::acc_zero(), gl::acc_zero()}; }
    static __device__ __forceinline__ void mul(A& s, gl::E2 x, gl::E2 y) {
        gl::acc_mul(s.s0, x.c0, y.c0);
        gl::acc_mul(s.s0, x.c1, gl::mul_small(y.c1, 7));
        gl::acc_mul(s.s1, x.c0, y.c1);
        gl::acc_mul(s.s1, x.c1, y.c0);
    }
    static __device__ __forceinline__ gl::E2 reduce(const A& s) {
        return gl::E2{gl::acc_reduce_wide(s.s0), gl::acc_reduce_wide(s.s1)};
    }
};

// Round polynomial of a product of D tables from D + 1 exact sums, one multiply-accumulate chain each per pair, reduced
// once at the end. Written a at 0, b at 1 and b - a as the leading coefficient (the value at infinity), the
// product of two tables takes three products (at 0, 1, infinity), and its other values are small combinations:
//   q(-1) = 2 q(0) + 2 q(inf) - q(1),   q(2) = 2 q(1) + 2 q(inf) - q(0).
//   D = 2: sums at 0, 1, infinity            D = 3: q times the third table at 0, 1, -1, infinity
//   D = 4: q times the other two's product at 0, 1, -1, 2, infinity
// Evaluating at 0 .. D takes (D + 1)(D - 1) reduced products and as many sums instead: eight against three reduced and
// four accumulated for D = 3 (2^22 almost-Goldilocks extension elements, first round: 168 -> 102 us), fifteen against six and five for D = 4.
template <class F, int D>
struct RoundSums {
    static_assert(D >= 2 && D <= 4, "see accumulate_pair for other counts");
    using T = typename F::T;
    using Sum = NarrowLazy<F>;
    typename Sum::A s[D + 1];
    static __device__ __forceinline__ T twice(T x) { return F::add(x, x); }
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int c = 0; c <= D; c++) s[c] = Sum::zero();
    }
    // lo, hi: the tables' values at 0 and 1
    __device__ __forceinline__ void add_pair(const T (&lo)[D], const T (&hi)[D]) {
        if constexpr (D == 2) {
            Sum::mul(s[0], lo[0], lo[1]);
            Sum::mul(s[1], hi[0], hi[1]);
            Sum::mul(s[2], F::sub(hi[0], lo[0]), F::sub(hi[1], lo[1]));
        } else {
            const T q0 = F::mul(lo[0], lo[1]), q1 = F::mul(hi[0], hi[1]);
            const T qi = F::mul(F::sub(hi[0], lo[0]), F::sub(hi[1], lo[1]));
            if constexpr (D == 3) {
                Sum::mul(s[0], q0, lo[2]);
                Sum::mul(s[1], q1, hi[2]);
                Sum::mul(s[2], F::sub(twice(F::add(q0, qi)), q1), F::sub(twice(lo[2]), hi[2]));
                Sum::mul(s[3], qi, F::sub(hi[2], lo[2]));
            } else {
                const T u0 = F::mul(lo[2], lo[3]), u1 = F::mul(hi[2], hi[3]);
                const T ui = F::mul(F::sub(hi[2], lo[2]), F::sub(hi[3], lo[3]));
                Sum::mul(s[0], q0, u0);
                Sum::mul(s[1], q1, u1);
                Sum::mul(s[2], F::sub(twice(F::add(q0, qi)), q1), F::sub(twice(F::add(u0, ui)), u1));
                Sum::mul(s[3], F::sub(twice(F::add(q1, qi)), q0), F::sub(twice(F::add(u1, ui)), u0));
                Sum::mul(s[4], qi, ui);
            }
        }
    }
    // acc[c] = this thread's share of P(c), c = 0 .. D; the values beyond the sums by differences of order D, which are
    // D! times the leading coefficient
    __device__ __forceinline__ void finish(T (&acc)[D + 1]) {
        T total[D + 1];
#pragma unroll
        for (int c = 0; c <= D; c++) total[c] = Sum::reduce(s[c]);
        acc[0] = total[0];
        acc[1] = total[1];
        if constexpr (D == 2) {
            acc[2] = F::sub(twice(F::add(total[1], total[2])), total[0]);
        } else if constexpr (D == 3) {
            const T c6 = twice(thrice(total[3]));
            acc[2] = F::add(F::add(thrice(F::sub(total[1], total[0])), total[2]), c6);
            acc[3] = F::add(F::add(thrice(F::sub(acc[2], total[1])), total[0]), c6);
        } else {
            const T c24 = twice(twice(twice(thrice(total[4]))));
            acc[2] = total[3];
            acc[3] = F::add(F::sub(step4(acc[2], acc[1], acc[0]), total[2]), c24);
            acc[4] = F::add(F::sub(step4(acc[3], acc[2], acc[1]), acc[0]), c24);
        }
    }

private:
    static __device__ __forceinline__ T thrice(T x) { return F::add(twice(x), x); }
    // 4 x - 6 y + 4 z
    static __device__ __forceinline__ T step4(T x, T y, T z) { return F::sub(twice(twice(F::add(x, z))), twice(thrice(y))); }
};

// ---- block-wide sum of NV residues per thread -------------------------------
// Warp shuffles, then one shared-memory hop across warps. Thread 0 writes the
// canonical totals to out[0..NV). blockDim.x must be a multiple of 32.
template <int NV, class AddFn, class CanonFn>
__device__ __forceinline__ void block_sum_store(uint64_t (&v)[NV], uint64_t* out, AddFn addf, CanonFn canonf) {
    __shared__ uint64_t sm[32][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = addf(v[k], __shfl_down_sync(0xffffffffu, v[k], off));
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) sm[warp][k] = v[k];
    }
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = lane < nw ? sm[lane][k] : 0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int k = 0; k < NV; k++) v[k] = addf(v[k], __shfl_down_sync(0xffffffffu, v[k], off));
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < NV; k++) out[k] = canonf(v[k]);
        }
    }
}

// acc[c] += prod_i (val_i + c * diff_i) for c = 0..D; consumes val.
template <class F, int D>
__device__ __forceinline__ void accumulate_pair(typename F::T (&val)[D], const typename F::T (&diff)[D],
                                                typename F::T (&acc)[D + 1]) {
#pragma unroll
    for (int c = 0; c <= D; c++) {
        typename F::T prod = val[0];
#pragma unroll
        for (int i = 1; i < D; i++) prod = F::mul(prod, val[i]);
        acc[c] = F::add(acc[c], prod);
        if (c < D) {
#pragma unroll
            for (int i = 0; i < D; i++) val[i] = F::add(val[i], diff[i]);
        }
    }
}

// Block partial -> global row; optionally the last block to finish adds all rows
// up ("last block done" pattern: a fence, one atomic ticket per block) and
// writes the (D+1)*NW canonical totals to final_out, so no second launch and no
// host-side summation is needed. `counter` must be zero on entry and is reset
// to zero by the last block. Rows written by other blocks are read with
// cache-global loads, which never hit a stale L1 line.
template <class F, int D>
__device__ __forceinline__ void store_partials(typename F::T (&acc)[D + 1], uint64_t* partial,
                                                unsigned int* counter, uint64_t* final_out) {
    constexpr int NV = (D + 1) * F::NW;
    uint64_t v[NV];
#pragma unroll
    for (int c = 0; c <= D; c++) F::to_words(acc[c], v + c * F::NW);
    block_sum_store<NV>(v, partial + (size_t)blockIdx.x * NV, typename F::WordAdd(), typename F::WordCanon());
    if (final_out == nullptr) return;
    __shared__ bool is_last;
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int ticket = atomicAdd(counter, 1u);
        is_last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = 0;
    for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = typename F::WordAdd()(v[k], __ldcg(partial + (size_t)b * NV + k));
    }
    block_sum_store<NV>(v, final_out, typename F::WordAdd(), typename F::WordCanon());
    if (threadIdx.x == 0) *counter = 0;
}

// Blocks per SM that the two kernels below keep registers for (RES). The exact sums of three and four tables want two. With
// seven and eight tables one block takes all 255 registers, which is faster while the grid has at most a block per SM; two
// blocks at 128, with some spills, are where it has more, and for the fold of eight tables, which spills either way. Measured,
// Goldilocks extension tables of 2^20, us at RES = 1 / 2: round message of eight, 148 blocks 231 / 340, 592 blocks 287 / 247;
// fold and message of seven (base tables) 119 / 147 and 161 / 133, of eight (extension) 315 / 283 and 349 / 214.
constexpr int blocks_resident(int d) { return d == 3 || d == 4 ? 2 : 1; }

// ---- round message ----------------------------------------------------------
// partial[(blockIdx.x * (D+1) + c) * NW ...] = this block's share of P(c).
template <class F, int D, int RES>
__global__ void __launch_bounds__(D == 2 ? 512 : 256, RES)   // exact sums in registers for D = 2, 3, 4
round_message_kernel(const uint64_t* __restrict__ polys, size_t stride, size_t half, uint64_t* __restrict__ partial,
                     unsigned int* counter, uint64_t* final_out) {
    using T = typename F::T;
    T acc[D + 1];
    const size_t step = (size_t)gridDim.x * blockDim.x;
    if constexpr (D >= 2 && D <= 4) {
        RoundSums<F, D> sums;
        sums.init();
        for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < half; y += step) {
            T lo[D], hi[D];
#pragma unroll
            for (int i = 0; i < D; i++) F::load2(polys + (size_t)i * stride * F::NW, 2 * y, lo[i], hi[i]);
            sums.add_pair(lo, hi);
        }
        sums.finish(acc);
    } else {
#pragma unroll
        for (int c = 0; c <= D; c++) acc[c] = F::zero();
        for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < half; y += step) {
            T val[D], diff[D];
#pragma unroll
            for (int i = 0; i < D; i++) {
                T a, b;
                F::load2(polys + (size_t)i * stride * F::NW, 2 * y, a, b);
                val[i] = a;
                diff[i] = F::sub(b, a);
            }
            accumulate_pair<F, D>(val, diff, acc);
        }
    }
    store_partials<F, D>(acc, partial, counter, final_out);
}

// ---- plain fold (out of place) ------------------------------------------------
// out[i*stride + y] = a + r (b - a); blockIdx.y selects the table.
template <class F>
__global__ void fold_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, typename F::T r,
                            size_t stride, size_t half) {
    using T = typename F::T;
    const uint64_t* pin = in + (size_t)blockIdx.y * stride * F::NW;
    uint64_t* pout = out + (size_t)blockIdx.y * stride * F::NW;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < half; y += step) {
        T a, b;
        F::load2(pin, 2 * y, a, b);
        F::store(pout, y, F::add(a, F::mul(r, F::sub(b, a))));
    }
}

// ---- fused fold + next message ---------------------------------------------------
// Input tables hold 4*quarter live elements each; the fold on r writes
// 2*quarter elements per table and the message of the following round is
// accumulated from them. FIn is the input field; the output and the message are
// always in FOut (a base-field input is lifted by the extension challenge).
template <class FIn, class FOut>
struct FoldOp;

template <class F>
struct FoldOp<F, F> {
    static __device__ __forceinline__ typename F::T apply(typename F::T a, typename F::T b, typename F::T r) {
        return F::add(a, F::mul(r, F::sub(b, a)));
    }
};
// Goldilocks: a + r (b - a) as two exact sums of products (the factor r with
// 7 r.c1 precomputed is loop invariant), one reduction per component.
template <>
struct FoldOp<GlBase, GlExt2> {
    static __device__ __forceinline__ gl::E2 apply(uint64_t a, uint64_t b, gl::E2 r) {
        return gl::e2_fma_pre_base(gl::e2_pre(r), gl::sub(b, a), a);
    }
};
template <>
struct FoldOp<GlExt2, GlExt2> {
    static __device__ __forceinline__ gl::E2 apply(gl::E2 a, gl::E2 b, gl::E2 r) {
        return gl::e2_fma_pre(gl::e2_pre(r), gl::e2_sub(b, a), a);
    }
};

template <class FIn, class FOut, int D, int RES>
__global__ void __launch_bounds__(BLOCK, RES)
fold_message_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, typename FOut::T r_val,
                    const uint64_t* __restrict__ r_ptr, size_t stride_in, size_t stride_out, size_t quarter,
                    uint64_t* __restrict__ partial, unsigned int* counter, uint64_t* final_out) {
    using TI = typename FIn::T;
    using TO = typename FOut::T;
    TO r = r_val;
    if (r_ptr != nullptr) r = FOut::load(r_ptr, 0);
    TO acc[D + 1];
    const size_t step = (size_t)gridDim.x * blockDim.x;
    if constexpr (D >= 2 && D <= 4) {
        RoundSums<FOut, D> sums;
        sums.init();
        for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < quarter; y += step) {
            TO lo[D], hi[D];
#pragma unroll
            for (int i = 0; i < D; i++) {
                TI e0, e1, e2, e3;
                const uint64_t* pin = in + (size_t)i * stride_in * FIn::NW;
                FIn::load2(pin, 4 * y, e0, e1);
                FIn::load2(pin, 4 * y + 2, e2, e3);
                lo[i] = FoldOp<FIn, FOut>::apply(e0, e1, r);
                hi[i] = FoldOp<FIn, FOut>::apply(e2, e3, r);
                FOut::store2(out + (size_t)i * stride_out * FOut::NW, 2 * y, lo[i], hi[i]);
            }
            sums.add_pair(lo, hi);
        }
        sums.finish(acc);
    } else {
#pragma unroll
        for (int c = 0; c <= D; c++) acc[c] = FOut::zero();
        for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < quarter; y += step) {
            TO val[D], diff[D];
#pragma unroll
            for (int i = 0; i < D; i++) {
                TI e0, e1, e2, e3;
                const uint64_t* pin = in + (size_t)i * stride_in * FIn::NW;
                FIn::load2(pin, 4 * y, e0, e1);
                FIn::load2(pin, 4 * y + 2, e2, e3);
                TO f0 = FoldOp<FIn, FOut>::apply(e0, e1, r);
                TO f1 = FoldOp<FIn, FOut>::apply(e2, e3, r);
                FOut::store2(out + (size_t)i * stride_out * FOut::NW, 2 * y, f0, f1);
                val[i] = f0;
                diff[i] = FOut::sub(f1, f0);
            }
            accumulate_pair<FOut, D>(val, diff, acc);
        }
    }
    store_partials<FOut, D>(acc, partial, counter, final_out);
}

// Last fold of a base-field table pair by an extension challenge (no message).
template <class FIn, class FOut>
__global__ void fold_lift_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, typename FOut::T r_val,
                                 const uint64_t* __restrict__ r_ptr, size_t stride_in, size_t stride_out, size_t half) {
    typename FOut::T r = r_val;
    if (r_ptr != nullptr) r = FOut::load(r_ptr, 0);
    const uint64_t* pin = in + (size_t)blockIdx.y * stride_in * FIn::NW;
    uint64_t* pout = out + (size_t)blockIdx.y * stride_out * FOut::NW;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < half; y += step) {
        typename FIn::T a, b;
        FIn::load2(pin, 2 * y, a, b);
        FOut::store(pout, y, FoldOp<FIn, FOut>::apply(a, b, r));
    }
}

}  // namespace sc
}  // namespace mb
