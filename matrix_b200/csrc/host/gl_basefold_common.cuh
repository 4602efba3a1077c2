// Shared by the single-GPU and the sharded Basefold host layers: device buffers, the kernels of the
// opening's inner sumcheck and query phase, the folding table and the commitment object.
//
//   BasefoldTable        goldilocks-cuda-rs/src/basefold.rs:267-362
//   DeviceMerkleTree     goldilocks-cuda-rs/src/merkle.rs:20-160
//   BasefoldCommitment   goldilocks-cuda-rs/src/basefold.rs:368-414 (commit_device)
#pragma once
#include <cstring>
#include <memory>
#include <atomic>
#include <vector>
#include "../basefold_kernels.cuh"
#include "../eq_kernels.cuh"
#include "../merkle_kernels.cuh"
#include "arrivals.hpp"
#include "host_tree_top.hpp"
#include "gl_transcript.hpp"
#include "pair_sumcheck.cuh"
#include "scratch_pool.hpp"

namespace mb {
namespace bf {
int evals_to_codeword_async(const uint64_t*, uint64_t*, uint64_t*, int, int, cudaStream_t);
int bit_reverse_async(const uint64_t*, uint64_t*, int, cudaStream_t);
}  // namespace bf
}  // namespace mb

using namespace mb;

namespace mbhost {

// ---- small RAII device buffer ----------------------------------------------------
struct DevBuf {
    uint64_t* p = nullptr;
    size_t words = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    int alloc(size_t w) {
        release();
        words = w;
        if (w == 0) return MB_OK;
        return pool_alloc(reinterpret_cast<void**>(&p), w * sizeof(uint64_t)) == cudaSuccess ? MB_OK : MB_ERR_CUDA;
    }
    void release() {
        pool_free(p);
        p = nullptr;
        words = 0;
    }
};

// ---- kernels private to the host layer ---------------------------------------------

// weights[k] = 1 / weights[k] for the (point, weight) table.
static __global__ void table_invert_kernel(uint64_t* table, size_t entries) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < entries; k += step)
        table[2 * k + 1] = gl::canon(gl::inv(table[2 * k + 1]));
}

// Oracle of the opening's inner sumcheck from tables in value form:
// with e = (eq[2j], eq[2j+1] - eq[2j]) and b likewise,
// c0 = sum e0 b0, c1 = sum (e0 b1 + e1 b0), c2 = sum e1 b1
// (the coefficients cuda/basefold.cuh:334-383 computes after its in-place
// interp step). BH_BASE: bh holds base-field values.
template <bool BH_BASE>
__device__ __forceinline__ void oracle_accumulate(gl::E2 q0, gl::E2 q1, gl::E2 b0, gl::E2 b1, gl::E2& a0, gl::E2& a1,
                                                  gl::E2& a2) {
    gl::E2 qd = gl::e2_sub(q1, q0), bd = gl::e2_sub(b1, b0);
    if (BH_BASE) {
        a0 = gl::e2_add(a0, gl::e2_mul_base(q0, b0.c0));
        a1 = gl::e2_add(a1, gl::e2_add(gl::e2_mul_base(q0, bd.c0), gl::e2_mul_base(qd, b0.c0)));
        a2 = gl::e2_add(a2, gl::e2_mul_base(qd, bd.c0));
    } else {
        a0 = gl::e2_add(a0, gl::e2_mul(q0, b0));
        a1 = gl::e2_add(a1, gl::e2_add(gl::e2_mul(q0, bd), gl::e2_mul(qd, b0)));
        a2 = gl::e2_add(a2, gl::e2_mul(qd, bd));
    }
}

// Block partials, then the last block to finish adds them up into final_out[6].
__device__ __forceinline__ void oracle_finish(gl::E2 a0, gl::E2 a1, gl::E2 a2, uint64_t* partial, unsigned int* counter,
                                              uint64_t* final_out) {
    uint64_t v[6] = {a0.c0, a0.c1, a1.c0, a1.c1, a2.c0, a2.c1};
    sc::block_sum_store<6>(v, partial + 6 * (size_t)blockIdx.x, sc::GlAdd(), sc::GlCanon());
    __shared__ bool is_last;
    if (threadIdx.x == 0) {
        __threadfence();
        is_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < 6; k++) v[k] = 0;
    for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < 6; k++) v[k] = gl::add(v[k], __ldcg(partial + 6 * (size_t)b + k));
    sc::block_sum_store<6>(v, final_out, sc::GlAdd(), sc::GlCanon());
    if (threadIdx.x == 0) *counter = 0;
}

// First oracle: eq (extension) x bh (base), both of length 2 * pairs.
static __global__ void __launch_bounds__(256)
oracle0_kernel(const uint64_t* __restrict__ eq, const uint64_t* __restrict__ bh, size_t pairs, uint64_t* partial,
               unsigned int* counter, uint64_t* final_out) {
    gl::E2 a0{0, 0}, a1{0, 0}, a2{0, 0};
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < pairs; j += step) {
        gl::E2 q0 = gl::e2_load(eq + 4 * j), q1 = gl::e2_load(eq + 4 * j + 2);
        ulonglong2 b = *reinterpret_cast<const ulonglong2*>(bh + 2 * j);
        oracle_accumulate<true>(q0, q1, gl::E2{b.x, 0}, gl::E2{b.y, 0}, a0, a1, a2);
    }
    oracle_finish(a0, a1, a2, partial, counter, final_out);
}

// One round: fold eq and bh on r (four inputs -> two outputs each) and
// accumulate the oracle of the folded tables. BH_BASE: bh_in is base field
// (round 0); outputs are always extension elements.
template <bool BH_BASE>
__global__ void __launch_bounds__(256)
open_round_kernel(const uint64_t* __restrict__ eq_in, const uint64_t* __restrict__ bh_in, gl::E2 r,
                  uint64_t* __restrict__ eq_out, uint64_t* __restrict__ bh_out, size_t quarter, uint64_t* partial,
                  unsigned int* counter, uint64_t* final_out) {
    gl::E2 a0{0, 0}, a1{0, 0}, a2{0, 0};
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t y = (size_t)blockIdx.x * blockDim.x + threadIdx.x; y < quarter; y += step) {
        const uint64_t* pe = eq_in + 8 * y;
        gl::E2 e0 = gl::e2_load(pe), e1 = gl::e2_load(pe + 2), e2 = gl::e2_load(pe + 4), e3 = gl::e2_load(pe + 6);
        gl::E2 q0 = gl::e2_add(e0, gl::e2_mul(r, gl::e2_sub(e1, e0)));
        gl::E2 q1 = gl::e2_add(e2, gl::e2_mul(r, gl::e2_sub(e3, e2)));
        gl::E2 b0, b1;
        if (BH_BASE) {
            ulonglong2 u = *reinterpret_cast<const ulonglong2*>(bh_in + 4 * y);
            ulonglong2 w = *reinterpret_cast<const ulonglong2*>(bh_in + 4 * y + 2);
            uint64_t d0 = gl::sub(u.y, u.x), d1 = gl::sub(w.y, w.x);
            b0 = gl::E2{gl::add(u.x, gl::mul(r.c0, d0)), gl::mul(r.c1, d0)};
            b1 = gl::E2{gl::add(w.x, gl::mul(r.c0, d1)), gl::mul(r.c1, d1)};
        } else {
            const uint64_t* pb = bh_in + 8 * y;
            gl::E2 f0 = gl::e2_load(pb), f1 = gl::e2_load(pb + 2), f2 = gl::e2_load(pb + 4), f3 = gl::e2_load(pb + 6);
            b0 = gl::e2_add(f0, gl::e2_mul(r, gl::e2_sub(f1, f0)));
            b1 = gl::e2_add(f2, gl::e2_mul(r, gl::e2_sub(f3, f2)));
        }
        q0 = gl::e2_canon(q0); q1 = gl::e2_canon(q1); b0 = gl::e2_canon(b0); b1 = gl::e2_canon(b1);
        gl::e2_store(eq_out + 4 * y, q0);
        gl::e2_store(eq_out + 4 * y + 2, q1);
        gl::e2_store(bh_out + 4 * y, b0);
        gl::e2_store(bh_out + 4 * y + 2, b1);
        oracle_accumulate<false>(q0, q1, b0, b1, a0, a1, a2);
    }
    oracle_finish(a0, a1, a2, partial, counter, final_out);
}

// ---- the opening's inner sumcheck, several rounds per pass --------------------------------------
// sum_x eq(t, x) bh(x) with eq factored (pair_kernels.cuh has the idea, here with one table): B rounds need the 2^B sums
//     S(m) = sum_s w(s) f(m, s)
// over the variables that are not among the next B. The table is the commitment's bit-reversed evaluations, in which the
// variable bound first is the top index bit: m and the challenges to fold select whole runs of the array, every access
// is coalesced, and the evaluations need not be put back into natural order. blockIdx.y = m. w(s) = WL[t] WH[h] for
// s = 256 h + t. Replaces an eq table, a reversed copy and one pass over both tables per round (1.1 ms of an opening at
// 2^24, and 10 us of every round of a small one).
struct OpenPassArgs {
    const uint64_t* in;      // 2^(v + fb) elements
    uint64_t* out;           // 2^v folded elements, or null
    int fb, v, rounds;       // challenges to fold; variables left after that; rounds of the next block
    const uint64_t *wl, *wh; // eq over the s variables: the low 8 (or fewer), and the others
    uint64_t* acc;           // [2^rounds][pr::grid_words(1)]
    uint64_t* sums;          // pinned: [2^rounds][2]
};
template <bool FOLD, bool BASE>
__global__ void __launch_bounds__(pr::BLK)
open_pass_kernel(const OpenPassArgs a, const __grid_constant__ pr::FoldWeights<pr::GlF> fw) {
    using F = pr::GlF;
    __shared__ gl::E2 sm[pr::BLK];
    chain_begin();
    const int t = threadIdx.x, m = blockIdx.y, sb = a.v - a.rounds;
    const size_t ns = (size_t)1 << sb, n = (size_t)1 << a.v;
    gl::Acc s0 = gl::acc_zero(), s1 = gl::acc_zero();
    gl::E2 x{0, 0};
    for (size_t h = blockIdx.x; h * pr::BLK < ns; h += gridDim.x) {
        const size_t s = h * pr::BLK + t;
        if (s >= ns) break;
        const size_t y = (size_t)m * ns + s;
        gl::E2 f;
        if constexpr (!FOLD) {
            f = BASE ? gl::E2{a.in[y], 0} : gl::e2_load(a.in + 2 * y);
        } else {
            gl::Acc c0 = gl::acc_zero(), c1 = gl::acc_zero();
#pragma unroll 4
            for (int j = 0; j < (1 << a.fb); j++) {
                const size_t i = ((size_t)j << a.v) + y;
                if (BASE) {
                    const uint64_t v = a.in[i];
                    gl::acc_mul(c0, fw.w[j].c0, v);
                    gl::acc_mul(c1, fw.w[j].c1, v);
                } else {
                    const gl::E2 v = gl::e2_load(a.in + 2 * i);
                    gl::acc_mul(c0, fw.w[j].c0, v.c0);
                    gl::acc_mul(c0, fw.w[j].c1w, v.c1);
                    gl::acc_mul(c1, fw.w[j].c0, v.c1);
                    gl::acc_mul(c1, fw.w[j].c1, v.c0);
                }
            }
            f = gl::e2_canon(gl::E2{gl::acc_reduce(c0), gl::acc_reduce(c1)});
            if (a.out != nullptr) gl::e2_store(a.out + 2 * y, f);
        }
        if (ns <= pr::BLK) {
            x = f;
        } else {
            const gl::E2Pre w = pr::load_weight<F>(a.wh + 4 * h);
            gl::acc_mul(s0, w.c0, f.c0);
            gl::acc_mul(s1, w.c1, f.c0);
            if constexpr (FOLD || !BASE) {
                gl::acc_mul(s0, w.c1w, f.c1);
                gl::acc_mul(s1, w.c0, f.c1);
            }
        }
    }
    if (ns > pr::BLK) x = gl::E2{gl::acc_reduce_wide(s0), gl::acc_reduce_wide(s1)};
    if (sb > 0 && (size_t)t < ns) x = F::fma(pr::load_weight<F>(a.wl + 4 * t), x, gl::E2{0, 0});
    gl::E2 total[1] = {x};
    chain_next();
    if (!pr::grid_sum<F, 1>(total, 0, sm, a.acc + pr::grid_words(1) * m)) return;
    if (t == 0) pr::store2(a.sums + 2 * m, sm[0].c0, sm[0].c1);
}

class OpenSumcheck {
public:
    using H = PairHost<pr::GlF, PairGl>;
    using E2 = gl::E2;
    // bh: 2^nv bit-reversed evaluations on the device; point: nv (c0, c1) pairs; sums: 32 words of pinned memory for the
    // passes' sums; acc: the scratch block's device words. Queues the first pass.
    int init(const uint64_t* bh, int nv, const uint64_t* point, uint64_t* sums, uint64_t* acc) {
        if (nv > pr::MAX_POINT) return MB_ERR_UNSUPPORTED;
        nv_ = nv; in_ = bh; sums_ = sums; acc_ = acc;
        pt_.resize(nv);
        r_.resize(nv);
        for (int i = 0; i < nv; i++) pt_[i] = H::canon(E2{point[2 * i], point[2 * i + 1]});
        const int parts = (nv + pr::MAX_B - 1) / pr::MAX_B;
        pr::TableSet set;
        int nt = 0;
        size_t words = 0;
        for (int i = 0, at = 0; i < parts; i++) {
            Stage s;
            s.first = at;
            s.rounds = (nv - at + (parts - i) - 1) / (parts - i);
            const int sb = nv - at - s.rounds, lo = sb < 8 ? sb : 8;   // index bit j of s goes with variable nv - 1 - j
            s.wl = words; set.d[nt].first = 0; set.d[nt].bits = lo; set.d[nt++].off = words; words += (size_t)4 << lo;
            s.wh = words; set.d[nt].first = lo; set.d[nt].bits = sb - lo; set.d[nt++].off = words; words += (size_t)4 << (sb - lo);
            stages_.push_back(s);
            at += s.rounds;
        }
        int rc = tabs_.alloc(words);
        if (rc != MB_OK) return rc;
        for (int i = 0; i < nv; i++) { set.pt[2 * i] = pt_[nv - 1 - i].c0; set.pt[2 * i + 1] = pt_[nv - 1 - i].c1; }
        {
            MB_KERNEL_ON("open_eq_tables", MB_STREAM);
            pr::eq_tables_kernel<pr::GlF><<<dim3(nt, pr::eq_table_chunks(set, nt)), pr::BLK, 0, MB_STREAM>>>(set, tabs_.p);
        }
        return pass();
    }
    // The sums of the pass queued last, if any, are there.
    int wait() const { return g_.empty() && stage_ < stages_.size() ? await_words(sums_, (size_t)2 << stages_[stage_].rounds) : MB_OK; }
    // The oracle of the current round, c0 c1 c2 (six words); after wait().
    void oracle(uint64_t* out6) {
        const Stage& st = stages_[stage_];
        if (g_.empty()) {
            const int B = st.rounds;
            g_.resize((size_t)1 << B);
            for (int m = 0; m < (1 << B); m++) {   // the top bit of m is the variable bound first
                int i = 0;
                for (int k = 0; k < B; k++) i |= ((m >> (B - 1 - k)) & 1) << k;
                g_[i] = E2{sums_[2 * m], sums_[2 * m + 1]};
            }
        }
        // eq of the block's later variables
        const int later = st.first + st.rounds - round_ - 1;
        E2 w[1 << pr::MAX_B];
        H::eq_vector(pt_.data() + round_ + 1, later, w);
        typename H::Dot da, db;
        for (int y = 0; y < (1 << later); y++) { da.mac(w[y], g_[2 * y]); db.mac(w[y], g_[2 * y + 1]); }
        const E2 a = da.value(), d = H::sub(db.value(), a), t = pt_[round_], one{1, 0};
        const E2 e0 = H::mul(scale_, H::sub(one, t)), e1 = H::mul(scale_, H::sub(H::add(t, t), one));
        const E2 c0 = H::mul(e0, a), c1 = H::add(H::mul(e0, d), H::mul(e1, a)), c2 = H::mul(e1, d);
        out6[0] = c0.c0; out6[1] = c0.c1; out6[2] = c1.c0; out6[3] = c1.c1; out6[4] = c2.c0; out6[5] = c2.c1;
    }
    int fold(E2 r) {
        const E2 t = pt_[round_], tr = H::mul(t, r);
        scale_ = H::mul(scale_, H::add(H::sub(H::sub(E2{1, 0}, t), r), H::add(tr, tr)));
        r_[round_++] = r;
        const Stage& st = stages_[stage_];
        if (round_ == st.first + st.rounds) {
            stage_++;
            g_.clear();
            return stage_ < stages_.size() ? pass() : MB_OK;
        }
        for (size_t y = 0; y < g_.size() / 2; y++) g_[y] = H::fold(g_[2 * y], g_[2 * y + 1], r);
        g_.resize(g_.size() / 2);
        return MB_OK;
    }

private:
    struct Stage {
        int first, rounds;
        size_t wl, wh;
    };
    static constexpr int GX = 148;   // blocks per sum at most: eight per SM with sixteen sums
    int pass() {
        const Stage& st = stages_[stage_];
        const int fb = stage_ ? stages_[stage_ - 1].rounds : 0;
        OpenPassArgs a;
        a.fb = fb; a.v = nv_ - st.first; a.rounds = st.rounds;
        a.wl = tabs_.p + st.wl; a.wh = tabs_.p + st.wh;
        a.acc = acc_; a.sums = sums_;
        expect_words(sums_, (size_t)2 << st.rounds);
        a.in = in_; a.out = nullptr;
        if (fb && stage_ + 1 < stages_.size()) {
            DevBuf& t = tables_[stage_ & 1];
            int rc = t.alloc((size_t)2 << a.v);
            if (rc != MB_OK) return rc;
            a.out = t.p;
        }
        pr::FoldWeights<pr::GlF> fw;
        if (fb) {   // index bit fb - 1 - k goes with challenge k
            E2 rev[pr::MAX_B], e[1 << pr::MAX_B];
            for (int k = 0; k < fb; k++) rev[k] = r_[st.first - 1 - k];
            H::eq_vector(rev, fb, e);
            for (int j = 0; j < (1 << fb); j++) fw.w[j] = gl::e2_pre(e[j]);
        }
        const size_t rows = (((size_t)1 << (a.v - a.rounds)) + pr::BLK - 1) / pr::BLK;
        const dim3 grid(rows < GX ? (unsigned)rows : GX, 1u << a.rounds);
        {
            MB_KERNEL_ON("open_pass", MB_STREAM);
            const auto k = !fb ? open_pass_kernel<false, true> : stage_ == 1 ? open_pass_kernel<true, true> : open_pass_kernel<true, false>;
            launch_chained(k, grid, pr::BLK, 0, MB_STREAM, a, fw);
        }
        if (a.out) in_ = a.out;
        return finish_async();
    }
    int nv_ = 0, round_ = 0;
    size_t stage_ = 0;
    const uint64_t* in_ = nullptr;
    uint64_t *sums_ = nullptr, *acc_ = nullptr;
    E2 scale_{1, 0};
    std::vector<Stage> stages_;
    std::vector<E2> pt_, r_, g_;
    DevBuf tabs_, tables_[2];
};

// Query phase: every value pair and authentication path of every query in
// one launch. Block q handles query q; out is the per-query part of the proof.
struct QueryLevels {
    int nv, lr;
    const uint64_t* commit_cw;    // base-field codeword
    const uint64_t* commit_tree;  // its tree
    const uint64_t* fcw[40];      // folded codewords (extension)
    const uint64_t* ftree[40];    // their trees
};

__device__ __forceinline__ void copy_path(const uint64_t* tree, size_t num_leaves, size_t leaf, uint64_t* out) {
    // layer l starts at 4 * (2 * num_leaves - (num_leaves >> (l - 1))) for l >= 1
    int depth = 0;
    for (size_t s = num_leaves; s > 1; s >>= 1) depth++;
    for (int t = threadIdx.x; t < depth * 4; t += blockDim.x) {
        int l = t >> 2, w = t & 3;
        size_t off = 2 * num_leaves - ((2 * num_leaves) >> l);  // digests before layer l
        size_t sib = (leaf >> l) ^ 1;
        out[t] = tree[4 * (off + sib) + w];
    }
}

static __global__ void query_gather_kernel(QueryLevels lv, const uint64_t* __restrict__ leaf_idx, uint64_t* __restrict__ out,
                                    size_t qwords) {
    const int nv = lv.nv, lr = lv.lr;
    uint64_t* pq = out + (size_t)blockIdx.x * qwords;
    const size_t leaf = (size_t)leaf_idx[blockIdx.x];
    uint64_t* vals = pq + 1;
    if (threadIdx.x == 0) {
        pq[0] = leaf;
        vals[0] = lv.commit_cw[2 * leaf];
        vals[1] = 0;
        vals[2] = lv.commit_cw[2 * leaf + 1];
        vals[3] = 0;
    }
    for (int t = threadIdx.x; t < (nv - 1) * 4; t += blockDim.x) {
        int i = t >> 2, w = t & 3;
        size_t idx = leaf >> (i + 1);
        vals[4 * (i + 1) + w] = lv.fcw[i][4 * idx + w];
    }
    uint64_t* pp = vals + 4 * nv;
    size_t leaves = (size_t)1 << (nv + lr - 1);
    copy_path(lv.commit_tree, leaves, leaf, pp);
    pp += 4 * (nv + lr - 1);
    for (int i = 0; i <= nv - 2; i++) {
        size_t fl = (size_t)1 << (nv + lr - 2 - i);
        copy_path(lv.ftree[i], fl, leaf >> (i + 1), pp);
        pp += 4 * (nv + lr - 2 - i);
    }
}

// ---- BasefoldTable ------------------------------------------------------------------
class BasefoldTable {
public:
    // basefold.rs:281-321: xorshift64 (13, 7, 17) mod p; x1 redrawn while equal
    // to x0; weight = 1 / (x1 - x0). The stream is sequential and runs on the
    // host; the inversions run on the device.
    int generate(int nv, int lr, int num_rounds, uint64_t seed) {
        if (nv < 1 || lr < 0 || num_rounds < 1 || num_rounds > nv || nv + lr > 34) return MB_ERR_ARG;
        num_vars = nv; log_rate = lr; rounds = num_rounds;
        level_offsets.clear(); level_sizes.clear();
        size_t total = 0;
        for (int i = 0; i < num_rounds; i++) {
            level_offsets.push_back(total);
            level_sizes.push_back((size_t)1 << (nv + lr - i - 1));
            total += level_sizes.back();
        }
        entries = total;
        uint64_t* h = nullptr;
        MB_CUDA(cudaMallocHost(&h, total * 2 * sizeof(uint64_t)));
        uint64_t s = seed;
        auto next = [&s]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s % gl::P; };
        for (size_t k = 0; k < total; k++) {
            uint64_t x0 = next(), x1 = next();
            while (x1 == x0) x1 = next();
            h[2 * k] = x0;
            h[2 * k + 1] = x1 >= x0 ? x1 - x0 : x1 + (gl::P - x0);
        }
        int rc = d_entries.alloc(total * 2);
        if (rc == MB_OK && cudaMemcpyAsync(d_entries.p, h, total * 2 * sizeof(uint64_t), cudaMemcpyHostToDevice,
                                           MB_STREAM) != cudaSuccess)
            rc = MB_ERR_CUDA;
        if (rc == MB_OK) {
            {
                MB_KERNEL_ON("table_invert", MB_STREAM);
                table_invert_kernel<<<grid_for(total, 256, 8), 256, 0, MB_STREAM>>>(d_entries.p, total);
            }
            // the levels that an opening folds on the host
            host_first = (size_t)num_rounds;
            while (host_first > 0 && level_sizes[host_first - 1] <= 2 * host_leaves(1)) host_first--;
            const size_t from = host_first < level_offsets.size() ? level_offsets[host_first] : total;
            host_entries.resize(2 * (total - from));
            if (!host_entries.empty() && cudaMemcpyAsync(host_entries.data(), d_entries.p + 2 * from, 8 * host_entries.size(), cudaMemcpyDeviceToHost,
                                                         MB_STREAM) != cudaSuccess)
                rc = MB_ERR_CUDA;
            const int done = finish_sync();
            if (rc == MB_OK) rc = done;
        }
        cudaFreeHost(h);
        return rc;
    }
    const uint64_t* device_level_ptr(int level) const { return d_entries.p + 2 * level_offsets[level]; }

    // the same in host memory, for levels of at most 2 host_leaves entries
    const uint64_t* host_level(int level) const { return host_entries.data() + 2 * (level_offsets[level] - level_offsets[host_first]); }

    int num_vars = 0, log_rate = 0, rounds = 0;
    size_t entries = 0, host_first = 0;
    std::vector<uint64_t> host_entries;
    std::vector<size_t> level_offsets, level_sizes;
    DevBuf d_entries;
};

// Merkle hash of commitments made from now on: 0 = Poseidon2, 1 = Monolith. The
// reference fixes this at build time (cargo feature "monolith", default on:
// goldilocks-cuda-rs/src/basefold.rs:11-14); a commitment remembers the hash it
// was built with and its openings use the same one.
inline std::atomic<int> g_merkle_hash{0};

// ---- BasefoldCommitment -----------------------------------------------------------------
class BasefoldCommitment {
public:
    // What the commitment keeps. Before anything that is given back once it is made (uploaded evaluations, scratch): those
    // leave no hole between it and what an opening takes. A large request that fits no free block makes the memory pool remap
    // its memory; with the scratch first, 2^24 from host memory took 30 ms or 40 ms to 1 s by turns.
    int allocate(int nv, int lr) {
        if (nv < 1 || lr < 0 || nv + lr > 32) return MB_ERR_ARG;
        num_vars = nv; log_rate = lr;
        const size_t cw_len = (size_t)1 << (nv + lr);
        int rc = d_bh_evals.alloc((size_t)1 << nv);
        if (rc == MB_OK) rc = d_codeword.alloc(cw_len);
        if (rc == MB_OK) rc = d_tree.alloc(4 * (cw_len - 1));
        return rc;
    }
    // commit_device (basefold.rs:382-414): interpolate, encode, Merkle tree. After allocate.
    int commit_device(const uint64_t* d_evals) {
        if (!d_evals) return MB_ERR_ARG;
        const int nv = num_vars, lr = log_rate;
        hash = g_merkle_hash.load();
        size_t n = (size_t)1 << nv, cw_len = (size_t)1 << (nv + lr);
        DevBuf work;
        int rc = work.alloc(n);
        if (rc != MB_OK) return rc;
        rc = bf::bit_reverse_async(d_evals, d_bh_evals.p, nv, MB_STREAM);
        if (rc == MB_OK) rc = bf::evals_to_codeword_async(d_evals, work.p, d_codeword.p, nv, lr, MB_STREAM);
        if (rc == MB_OK)
            rc = hash ? mk::build_tree_periodic<mk::HashMonolith>(d_codeword.p, d_tree.p, cw_len / 2, (size_t)1 << lr, MB_STREAM)
                      : mk::build_tree_periodic<mk::HashPoseidon2>(d_codeword.p, d_tree.p, cw_len / 2, (size_t)1 << lr, MB_STREAM);
        if (rc != MB_OK) return rc;
        MB_CUDA(cudaMemcpyAsync(root, d_tree.p + 4 * (cw_len - 2), 32, cudaMemcpyDeviceToHost, MB_STREAM));
        MB_CUDA(cudaStreamSynchronize(MB_STREAM));
        return MB_OK;
    }
    uint64_t root[4] = {0, 0, 0, 0};
    int num_vars = 0, log_rate = 0, hash = 0;
    DevBuf d_codeword, d_bh_evals, d_tree;
};

// ---- host hashing of tree tops: host_tree_top.hpp -------------------------------------------
// A scratch block for the length of a scope (nothing may still be writing it when the scope ends).
struct ScopedScratch {
    ScratchBlock b = ScratchPool::take();
    uint64_t* p = b.host;
    ScopedScratch() = default;
    ScopedScratch(const ScopedScratch&) = delete;
    ScopedScratch& operator=(const ScopedScratch&) = delete;
    ~ScopedScratch() {
        if (b) ScratchPool::give(b, cudaStreamSynchronize(MB_STREAM) == cudaSuccess);
    }
};

// One round's codeword fold and the tree over the folded codeword, queued; the layer of min(leaves, host_top) digests
// goes to `nodes` (pinned). f: source, table level, target and challenge of the fold; mixed: the source is base field.
inline int queue_fold_tree(int hash, bool mixed, const mk::FoldSource& f, uint64_t* d_tree, size_t leaves, uint64_t* nodes) {
    const size_t stop = host_top(hash);
    if (hash)
        return mixed ? mk::fold_tree<mk::HashMonolith, true>(f, d_tree, leaves, MB_STREAM, nodes, stop)
                     : mk::fold_tree<mk::HashMonolith, false>(f, d_tree, leaves, MB_STREAM, nodes, stop);
    return mixed ? mk::fold_tree<mk::HashPoseidon2, true>(f, d_tree, leaves, MB_STREAM, nodes, stop)
                 : mk::fold_tree<mk::HashPoseidon2, false>(f, d_tree, leaves, MB_STREAM, nodes, stop);
}

// nodes: the layer of `count` digests (a power of two, at most HOST_TOP) the device left; upper: pinned staging for
// count - 1 digests that stays untouched until the stream has run the upload; d_tree: the tree of num_leaves
// leaves (2 num_leaves - 1 digests, layers back to back). root receives the root.
inline int host_finish_top(int hash, const uint64_t* nodes, size_t count, uint64_t* upper, uint64_t* d_tree, size_t num_leaves,
                           uint64_t* root, cudaStream_t st) {
    host_hash_top(hash, nodes, count, upper, root);
    if (count > 1)
        MB_CUDA(cudaMemcpyAsync(d_tree + 4 * (2 * num_leaves - count), upper, 32 * (count - 1), cudaMemcpyHostToDevice, st));
    return MB_OK;
}

// Pinned staging of the calling thread, grown on demand (contents are not kept across a growth).
inline uint64_t* pinned_arena(size_t words) {
    struct Holder {
        uint64_t* p = nullptr;
        size_t cap = 0;
        ~Holder() { if (p) cudaFreeHost(p); }
    };
    static thread_local Holder h;
    if (h.cap < words) {
        if (h.p) cudaFreeHost(h.p);
        h.p = nullptr;
        h.cap = 0;
        if (cudaMallocHost(&h.p, words * sizeof(uint64_t)) != cudaSuccess) { h.p = nullptr; return nullptr; }
        h.cap = words;
    }
    return h.p;
}

inline size_t query_words(int nv, int lr) {
    size_t w = 1 + (size_t)nv * 4 + 4 * (size_t)(nv + lr - 1);
    for (int i = 0; i <= nv - 2; i++) w += 4 * (size_t)(nv + lr - 2 - i);
    return w;
}
inline size_t proof_words(int nv, int lr, int nq) {
    return 2 + (size_t)nv * 6 + (size_t)(nv - 1) * 4 + ((size_t)2 << lr) + (size_t)nq * query_words(nv, lr);
}

}  // namespace mbhost
