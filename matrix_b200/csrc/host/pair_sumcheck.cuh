// Host side of the several-rounds-per-pass sumcheck over products of two tables (pair_kernels.cuh, pair_mma_kernels.cuh):
//     sum_x w(x) sum_k s_k a_k(x) b_k(x),   w = 1 or eq(t, x) on the first eq_vars variables,
// for K instances whose factors s_k may be chosen after the first pass (powers of a challenge). The object plans the
// blocks of rounds, queues the passes and runs the rounds of a block on the matrices they return; the last rounds, on
// tables of at most 512 elements together, run on the host altogether. The caller owns the transcript.
//
//   tensor cores      passes over 2^14 elements and more, three rounds each, four on words of the base field: their products
//                     cost next to nothing there (a pass that folds words to 2^16 elements takes 15 us, 26 without; 2^11 and fewer
//                     elements a table are less than a tile).
//   rounds per block  otherwise 4: a round more doubles the products per element (2^B), which pays while a launch and a
//                     synchronisation or wait (9 to 12 us) cost more than they do, and with at most 64 instances these passes have at
//                     most 2^17 elements. In every case bounded by what the host then has to fold, K 4^B entries.
//   host tables       2^t elements per table with K 2^t <= 512: the rest of a proof on them takes a core about as long
//                     as one more pass and its synchronisation.
//   all on the host   base-field tables of at most 2^10 elements: the copy and the rounds (35 us) cost less than two passes.
#pragma once
#include <vector>
#include "../common.cuh"
#include "../pair_kernels.cuh"
#include "../pair_mma_kernels.cuh"
#include "arrivals.hpp"
#include "host_field.hpp"
#include "scratch_pool.hpp"

namespace mbhost {

using namespace mb;

// Host arithmetic by field: canonical words in and out.
struct PairGl : hf::GlE2Ops {
    static constexpr uint64_t TOP = 0xFFFFFFFE00000001ULL;                       // 2^128 mod p = -2^32 mod p
};
struct PairAgl : hf::AglE2Ops {
    static constexpr uint64_t TOP = 63ULL * (1ULL << 32) + 992ULL;               // 2^128 mod q
};
template <class F, class O>
struct PairHost {
    using E2 = typename F::E2;
    static E2 mul(E2 a, E2 b) {
        E2 r;
        hf::e2_mul<O>(a.c0, a.c1, b.c0, b.c1, r.c0, r.c1);
        return r;
    }
    static E2 add(E2 a, E2 b) { return E2{O::add(a.c0, b.c0), O::add(a.c1, b.c1)}; }
    static E2 sub(E2 a, E2 b) { return E2{O::sub(a.c0, b.c0), O::sub(a.c1, b.c1)}; }
    static E2 fold(E2 a, E2 b, E2 r) { return add(a, mul(r, sub(b, a))); }
    static E2 canon(E2 a) { return E2{O::canon(a.c0), O::canon(a.c1)}; }
    // sum of products, reduced once
    struct Wide {
        hf::u128 s = 0;
        uint64_t top = 0;
        void mac(uint64_t x, uint64_t y) {
            const hf::u128 p = (hf::u128)x * y;
            s += p;
            top += s < p;
        }
        uint64_t red() const { return O::red((hf::u128)top * O::TOP + O::red(s)); }
    };
    struct Dot {
        Wide p00, p11, p01;
        void mac(E2 a, E2 b) {
            p00.mac(a.c0, b.c0);
            p11.mac(a.c1, b.c1);
            p01.mac(a.c0, b.c1);
            p01.mac(a.c1, b.c0);
        }
        E2 value() const { return E2{O::canon(O::red((hf::u128)p11.red() * O::W + p00.red())), O::canon(p01.red())}; }
    };
    // out[x] = prod_j (x_j ? r_j : 1 - r_j)
    static void eq_vector(const E2* r, int n, E2* out) {
        out[0] = E2{1, 0};
        for (int b = 0; b < n; b++)
            for (int x = 0; x < (1 << b); x++) {
                const E2 hi = mul(out[x], r[b]);
                out[x + (1 << b)] = hi;
                out[x] = sub(out[x], hi);
            }
    }
};

template <class F, class O>
class PairSumcheck {
public:
    using H = PairHost<F, O>;
    using E2 = typename F::E2;
    ~PairSumcheck() {
        if (scratch_) {   // nothing may still be writing it
            const bool clean = cudaStreamSynchronize(MB_STREAM) == cudaSuccess;
            ScratchPool::give(scratch_, clean && bad_ == MB_OK && pin_[ERROR_WORD] == 0);
        }
        pool_free(t0_);
        pool_free(t1_);
        pool_free(tabs_);
    }
    // a, b: instance 0's device tables of 2^n elements (never written), instances inst_stride words apart; base: base
    // field words, else (c0, c1). eq_pt: host, eq_vars (c0, c1) pairs, or null. Queues the first pass.
    int init(const uint64_t* a, const uint64_t* b, size_t inst_stride, int K, int n, bool base, const uint64_t* eq_pt, int eq_vars) {
        a_ = a; b_ = b; stride_ = inst_stride; K_ = K; n_ = n; base_ = base;
        pt_.resize(eq_vars);
        for (int i = 0; i < eq_vars; i++) pt_[i] = H::canon(E2{eq_pt[2 * i], eq_pt[2 * i + 1]});
        int t = 0;
        while (t < 9 && ((size_t)K << (t + 1)) <= 512) t++;
        if (base && ((size_t)K << n) <= 1024 && n > t) t = n;
        for (int v = n; v > t;) {
            const size_t size = (size_t)K << v;
            const bool first = v == n, words = base && blocks_.size() <= 1;   // a pass over words of the base field
            const int fb = first ? 0 : blocks_.back().rounds;
            const bool mma = size >= MMA_MIN && v >= pr::mma_min_vars(fb > 0, words) && (first || pr::mma_folds(fb, words));
            int g = mma ? (first && base ? 4 : 3) : 4;
            while (g > 1 && ((size_t)K << (2 * g)) > 1024) g--;
            if (g > v - t) g = v - t;
            blocks_.push_back(Block{n - v, g, 0, 0, 0, 63, 0, mma});
            v -= g;
        }
        tail_first_ = n - (n > t ? t : n);
        scratch_ = ScratchPool::take();
        if (!scratch_) return MB_ERR_CUDA;
        pin_ = scratch_.host;
        pin_[ERROR_WORD] = 0;
        r_.resize(n);
        cap_ = sm_count() * 4 / K > 1 ? sm_count() * 4 / K : 1;   // a wave: four blocks of at most 64 registers fit an SM
        int rc = tables();
        if (rc == MB_OK) rc = pass();
        // what the later passes fold into, allocated while the first one runs
        for (size_t i = 1; rc == MB_OK && i < blocks_.size() && i <= 2; i++)
            if (pool_alloc((void**)(i == 1 ? &t0_ : &t1_), sizeof(uint64_t) * ((size_t)4 << (n - blocks_[i].first)) * K) != cudaSuccess)
                rc = MB_ERR_CUDA;
        return failed(rc);
    }
    // The instances' factors (K = 1: not needed). sums() and fold() may be called from then on; before the first fold the
    // factors may be replaced.
    int set_scale(const E2* s) {
        scale_.assign(s, s + K_);
        m_.clear();
        return MB_OK;
    }
    // sum_x w(x) a_k(x) b_k(x) of every instance, before the first fold
    int claims(E2* out) {
        int rc = wait();
        if (rc != MB_OK) return rc;
        if (host_) {
            suffix(0, n_);
            for (int k = 0; k < K_; k++) out[k] = total(k);
            return MB_OK;
        }
        const int g = blocks_[0].rounds, G = 1 << g;
        std::vector<E2> w(G, E2{1, 0});
        const int we = (int)pt_.size() < g ? (int)pt_.size() : g;
        if (we) H::eq_vector(pt_.data(), we, w.data());
        for (int x = 1 << we; x < G; x++) w[x] = w[x & ((1 << we) - 1)];
        for (int k = 0; k < K_; k++) {
            typename H::Dot d;
            for (int m = 0; m < G; m++) d.mac(w[m], entry(k, m, m));
            out[k] = d.value();
        }
        return MB_OK;
    }
    // T(0), T(1) and the leading coefficient of this round's sum without the round's own eq factor: the round polynomial
    // is eq_scale() ((1 - t)(1 - c) + t c) T(c) while the round is below eq_vars, eq_scale() T(c) from then on.
    int sums(E2& s0, E2& s1, E2& s2) {
        int rc = wait();
        if (rc != MB_OK) return rc;
        if (host_) { host_sums(s0, s1, s2); return MB_OK; }
        if (m_.empty()) combine();
        const int half = side_ / 2;
        s0 = s1 = E2{0, 0};
        E2 cross{0, 0};
        if (half > 1 && weighted_) {
            typename H::Dot d0, d1, dc;
            const E2* w = weights(half);
            for (int m = 0; m < half; m++) {
                d0.mac(w[m], at(2 * m, 2 * m));
                d1.mac(w[m], at(2 * m + 1, 2 * m + 1));
                dc.mac(w[m], H::add(at(2 * m, 2 * m + 1), at(2 * m + 1, 2 * m)));
            }
            s0 = d0.value(); s1 = d1.value(); cross = dc.value();
        } else {
            for (int m = 0; m < half; m++) {
                s0 = H::add(s0, at(2 * m, 2 * m));
                s1 = H::add(s1, at(2 * m + 1, 2 * m + 1));
                cross = H::add(cross, H::add(at(2 * m, 2 * m + 1), at(2 * m + 1, 2 * m)));
            }
        }
        s2 = H::sub(H::add(s0, s1), cross);
        return MB_OK;
    }
    // Stands on its own: the round's sums need not have been asked for.
    int fold(E2 r) {
        int rc = wait();   // the rounds may be the host's by now
        if (rc != MB_OK) return rc;
        const int round = round_++;
        r_[round] = r;
        if (round < (int)pt_.size()) {
            const E2 t = pt_[round], tr = H::mul(t, r);   // (1 - t)(1 - r) + t r = 1 - t - r + 2 t r
            eq_scale_ = H::mul(eq_scale_, H::add(H::sub(H::sub(E2{1, 0}, t), r), H::add(tr, tr)));
        }
        if (host_) { host_fold(r); return MB_OK; }
        const Block& bl = blocks_[block_];
        if (round + 1 == bl.first + bl.rounds) {
            block_++;
            return failed(pass());
        }
        if (m_.empty()) combine();
        const int half = side_ / 2;   // rows, then columns
        for (int i = 0; i < half; i++)
            for (int j = 0; j < side_; j++) at(i, j) = H::fold(at(2 * i, j), at(2 * i + 1, j), r);
        for (int i = 0; i < half; i++)
            for (int j = 0; j < half; j++) at(i, j) = H::fold(at(i, 2 * j), at(i, 2 * j + 1), r);
        side_ = half;
        return MB_OK;
    }
    // a_k(R), b_k(R) after the last fold
    int finals(E2* a, E2* b) {
        int rc = wait();
        if (rc != MB_OK) return rc;
        for (int k = 0; k < K_; k++) { a[k] = ta_[(size_t)k * tn_]; b[k] = tb_[(size_t)k * tn_]; }
        return MB_OK;
    }
    E2 eq_scale() const { return eq_scale_; }
    E2 eq_coord(int round) const { return pt_[round]; }

private:
    static constexpr size_t ERROR_WORD = ScratchPool::WORDS - 2;
    static constexpr size_t MMA_MIN = (size_t)1 << 14;
    // Folds of at most this many tiles of 256 elements, over all instances: pair_small_kernel. Limits of 32 to 128 measure the same (all
    // rounds of three instances of 2^15: 168 us; of five of 2^14: 165), 16 and 256 one or two per cent more (172 and 170, 168 and 167).
    static constexpr size_t SMALL_TILES = 64;
    struct Block {
        int first, rounds;
        size_t wl, wh;      // word offsets of the eq tables
        int lo, row_shift;
        size_t row_mask;
        bool mma;           // on the tensor cores
    };
    // eq tables of the passes: over the variables above a block, those of WL first
    int tables() {
        const int ne = (int)pt_.size();
        pr::TableSet set;
        int nt = 0;
        size_t words = 0;
        const auto table = [&](int first, int bits) {
            set.d[nt].first = first;
            set.d[nt].bits = bits;
            set.d[nt].off = words;
            words += (size_t)4 << bits;
            return set.d[nt++].off;
        };
        for (Block& b : blocks_) {
            const int above = ne - b.first - b.rounds;
            if (above <= 0) continue;
            const int most = b.mma ? pr::MMA_ROW_BITS : pr::ROW_BITS;
            b.lo = above < most ? above : most;
            b.wl = table(b.first + b.rounds, b.lo);
            b.wh = table(b.first + b.rounds + b.lo, above - b.lo);
            if (above > b.lo) {
                b.row_shift = b.lo + b.rounds;
                b.row_mask = ((size_t)1 << (above - b.lo)) - 1;
            }
        }
        if (!nt) return MB_OK;
        if (ne > pr::MAX_POINT) return MB_ERR_UNSUPPORTED;
        MB_CUDA(pool_alloc((void**)&tabs_, sizeof(uint64_t) * words));
        for (int i = 0; i < ne; i++) { set.pt[2 * i] = pt_[i].c0; set.pt[2 * i + 1] = pt_[i].c1; }
        MB_KERNEL("pair_eq_tables");
        pr::eq_tables_kernel<F><<<dim3(nt, pr::eq_table_chunks(set, nt)), pr::BLK, 0, MB_STREAM>>>(set, tabs_);
        return finish_async();
    }
    // The pass before block block_ (or, after the last one, before the host tables): folds the challenges of the block
    // before and queues the matrices of this one.
    int pass() {
        const int from = block_ > 0 ? blocks_[block_ - 1].first : 0, fb = block_ > 0 ? blocks_[block_ - 1].rounds : 0;
        const bool last = block_ == blocks_.size();
        pr::FoldWeights<F> fw;
        E2 e[1 << pr::MAX_B];
        H::eq_vector(r_.data() + from, fb, e);
        for (int i = 0; i < (1 << fb); i++)
            fw.w[i] = typename F::Pre{e[i].c0, e[i].c1, O::canon(O::red((hf::u128)e[i].c1 * O::W))};
        pr::PairArgs p{};
        p.fb = fb;
        p.a = a_; p.b = b_; p.in_stride = stride_;
        p.v = n_ - (last ? tail_first_ : blocks_[block_].first);
        if (last) {
            p.out = pin_;
            tn_ = (size_t)1 << p.v;
            if (fb == 0) return copy_tables();   // everything on the host
        } else if (fb) {
            p.out = flip_ ? t1_ : t0_;
            flip_ = !flip_;
        }
        const int gb = last ? 0 : blocks_[block_].rounds;
        bool weighted = false;
        if (!last) {
            const Block& b = blocks_[block_];
            weighted = (int)pt_.size() > b.first + b.rounds;
            p.lo = b.lo; p.row_shift = b.row_shift; p.row_mask = b.row_mask;
            p.wl = tabs_ + b.wl; p.wh = tabs_ + b.wh;
        }
        p.acc = scratch_.dev; p.sums = pin_;
        arriving_ = 2 * (size_t)K_ * (last ? 2 * tn_ : (size_t)1 << (2 * gb));
        expect_words(pin_, arriving_);
        if (!last && blocks_[block_].mma) {
            int rc = launch_mma(gb, weighted, p, fw);
            if (rc != MB_OK) return rc;
        } else {
            const size_t n = (size_t)1 << p.v, tiles = (n + pr::BLK - 1) / pr::BLK;
            if (fb && tiles * K_ <= SMALL_TILES) {
                // threads an element: as many as have two inputs each and leave half as many blocks as SMs (with as many as
                // SMs the blocks' atomics on the same sums take longer than the products saved: 2^20 elements 282 -> 280 us a proof)
                int s = 0;
                while (s + 1 < fb && (n << (s + 1)) / (pr::BLK / 2) * K_ <= (size_t)sm_count() / 2) s++;
                const size_t tile = (pr::BLK / 2) >> s;
                const dim3 few((unsigned)((n + tile - 1) / tile), K_);
                MB_KERNEL("pair_small");
                base_ ? launch_small<true>(gb, weighted, few, p, s, fw) : launch_small<false>(gb, weighted, few, p, s, fw);
            } else {
                const dim3 grid(tiles < (size_t)cap_ ? (unsigned)tiles : (unsigned)cap_, K_);
                MB_KERNEL("pair_pass");
                if (fb) base_ ? launch<true, true>(gb, weighted, grid, p, fw) : launch<true, false>(gb, weighted, grid, p, fw);
                else base_ ? launch<false, true>(gb, weighted, grid, p, fw) : launch<false, false>(gb, weighted, grid, p, fw);
            }
        }
        if (p.out && !last) {   // the folded tables are the next pass's input
            a_ = p.out;
            b_ = p.out + ((size_t)2 << p.v);
            stride_ = (size_t)4 << p.v;
        }
        if (fb) base_ = false;
        pending_ = true;
        m_.clear();
        return finish_async();
    }
    template <bool FOLD, bool BASE, int GB>
    static void launch_w(bool weighted, dim3 grid, const pr::PairArgs& p, const pr::FoldWeights<F>& fw) {
        if (weighted) pr::pair_pass_kernel<F, FOLD, GB, BASE, true><<<grid, pr::BLK, sizeof(uint64_t) * ((size_t)3 << p.lo), MB_STREAM>>>(p, fw);
        else pr::pair_pass_kernel<F, FOLD, GB, BASE, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
    }
    template <bool FOLD, bool BASE>
    static void launch(int gb, bool weighted, dim3 grid, const pr::PairArgs& p, const pr::FoldWeights<F>& fw) {
        switch (gb) {
            case 0: pr::pair_pass_kernel<F, true, 0, BASE, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw); break;
            case 1: launch_w<FOLD, BASE, 1>(weighted, grid, p, fw); break;
            case 2: launch_w<FOLD, BASE, 2>(weighted, grid, p, fw); break;
            case 3: launch_w<FOLD, BASE, 3>(weighted, grid, p, fw); break;
            default: launch_w<FOLD, BASE, 4>(weighted, grid, p, fw); break;
        }
    }
    template <bool BASE, int GB>
    static void launch_small_w(bool weighted, dim3 grid, const pr::PairArgs& p, int s, const pr::FoldWeights<F>& fw) {
        if (weighted) pr::pair_small_kernel<F, GB, BASE, true><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
        else pr::pair_small_kernel<F, GB, BASE, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
    }
    template <bool BASE>
    static void launch_small(int gb, bool weighted, dim3 grid, const pr::PairArgs& p, int s, const pr::FoldWeights<F>& fw) {
        switch (gb) {
            case 0: launch_small_w<BASE, 0>(false, grid, p, s, fw); break;
            case 1: launch_small_w<BASE, 1>(weighted, grid, p, s, fw); break;
            case 2: launch_small_w<BASE, 2>(weighted, grid, p, s, fw); break;
            case 3: launch_small_w<BASE, 3>(weighted, grid, p, s, fw); break;
            default: launch_small_w<BASE, 4>(weighted, grid, p, s, fw); break;
        }
    }
    template <bool FOLD, bool BASE, bool WEIGHTED>
    static int launch_mma_as(dim3 grid, uint32_t smem, const pr::PairMmaArgs& p, const pr::FoldWeights<F>& fw) {
        const auto k = pr::pair_mma_kernel<F, FOLD, BASE, WEIGHTED>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return MB_ERR_CUDA;
        k<<<grid, pr::MMA_BLK, smem, MB_STREAM>>>(p, fw);
        return MB_OK;
    }
    // one block an SM, shared out over the instances
    int launch_mma(int gb, bool weighted, const pr::PairArgs& q, const pr::FoldWeights<F>& fw) {
        pr::PairMmaArgs p{};
        p.fb = q.fb; p.a = q.a; p.b = q.b; p.in_stride = q.in_stride; p.out = q.out; p.v = q.v; p.g = gb;
        p.lo = q.lo; p.row_shift = q.row_shift; p.row_mask = q.row_mask; p.wl = q.wl; p.wh = q.wh;
        p.acc = q.acc; p.sums = q.sums; p.error = pin_ + ERROR_WORD;
        const size_t tile = q.fb ? pr::MMA_FOLD_TILE : pr::MMA_RAW_ROWS * (base_ ? 16 : 8), tiles = ((size_t)1 << q.v) / tile;
        const size_t most = sm_count() / K_ > 1 ? sm_count() / K_ : 1;
        const dim3 grid(tiles < most ? (unsigned)tiles : (unsigned)most, K_);
        MB_KERNEL("pair_mma");
        if (q.fb) {
            const uint32_t smem = pr::mma_fold_smem(base_ ? 4 - q.fb : 3 - q.fb);
            if (weighted) return base_ ? launch_mma_as<true, true, true>(grid, smem, p, fw) : launch_mma_as<true, false, true>(grid, smem, p, fw);
            return base_ ? launch_mma_as<true, true, false>(grid, smem, p, fw) : launch_mma_as<true, false, false>(grid, smem, p, fw);
        }
        const uint32_t smem = pr::mma_raw_smem(base_, weighted);
        if (weighted) return base_ ? launch_mma_as<false, true, true>(grid, smem, p, fw) : launch_mma_as<false, false, true>(grid, smem, p, fw);
        return base_ ? launch_mma_as<false, true, false>(grid, smem, p, fw) : launch_mma_as<false, false, false>(grid, smem, p, fw);
    }
    int copy_tables() {
        const size_t w = tn_ * (base_ ? 1 : 2);
        if (2 * w * K_ > ScratchPool::WORDS) return MB_ERR_UNSUPPORTED;
        pending_ = true;
        arriving_ = 2 * w * K_;
        expect_words(pin_, arriving_);
        MB_KERNEL("pair_tables");
        pr::send_tables_kernel<F><<<dim3((unsigned)((w + pr::BLK - 1) / pr::BLK), 2 * K_), pr::BLK, 0, MB_STREAM>>>(a_, b_, stride_, w, pin_);
        return finish_async();
    }
    // A pass that could not be queued or did not finish leaves nothing to go on from: every later call returns its error too.
    int failed(int rc) {
        if (rc != MB_OK) bad_ = rc;
        return rc;
    }
    // Results of the pass queued last.
    int wait() {
        if (bad_ != MB_OK || !pending_) return bad_;
        if (await_words(pin_, arriving_) != MB_OK) return failed(MB_ERR_CUDA);
        pending_ = false;
        if (pin_[ERROR_WORD] != 0) return failed(MB_ERR_CUDA);   // a wait of a pass on the tensor cores ran out
        if (block_ < blocks_.size()) return MB_OK;
        host_ = true;
        const size_t nw = base_ ? 1 : 2;
        ta_.resize(tn_ * K_);
        tb_.resize(tn_ * K_);
        for (int k = 0; k < K_; k++)
            for (size_t x = 0; x < tn_; x++) {
                const uint64_t *p = pin_ + ((2 * (size_t)k) * tn_ + x) * nw, *q = p + tn_ * nw;
                ta_[k * tn_ + x] = H::canon(E2{p[0], nw == 2 ? p[1] : 0});
                tb_[k * tn_ + x] = H::canon(E2{q[0], nw == 2 ? q[1] : 0});
            }
        live_ = tn_;
        words_ = nw == 1;
        return MB_OK;
    }
    // ---- the rounds of a block on the matrix ----
    E2 entry(int k, int i, int j) const {
        const int g = blocks_[block_].rounds;
        const uint64_t* p = pin_ + 2 * (((size_t)k << (2 * g)) + ((size_t)i << g) + j);
        return E2{p[0], p[1]};
    }
    E2& at(int i, int j) { return m_[(size_t)i * width_ + j]; }
    void combine() {
        const Block& b = blocks_[block_];
        side_ = width_ = 1 << b.rounds;
        m_.resize((size_t)width_ * width_);
        for (int i = 0; i < width_; i++)
            for (int j = 0; j < width_; j++) {
                if (scale_.empty()) {
                    at(i, j) = entry(0, i, j);
                } else {
                    typename H::Dot d;
                    for (int k = 0; k < K_; k++) d.mac(scale_[k], entry(k, i, j));
                    at(i, j) = d.value();
                }
            }
        weighted_ = (int)pt_.size() > b.first + 1;
        if (weighted_) suffix(b.first, b.first + b.rounds);
    }
    // eq over the variables above each round of [first, last): for round last - 1 one entry, then 2, 4, .. , back to
    // back; variables without a coordinate weigh 1
    void suffix(int first, int last) {
        w_.assign((size_t)1 << (last - first), E2{1, 0});
        size_t at = 0;
        for (int j = last - 2; j >= first; j--) {
            const size_t n = (size_t)1 << (last - 2 - j);
            const bool has = j + 1 < (int)pt_.size();
            for (size_t y = 0; y < n; y++) {
                const E2 lo = w_[at + y], hi = has ? H::mul(lo, pt_[j + 1]) : lo;
                w_[at + n + 2 * y] = has ? H::sub(lo, hi) : lo;
                w_[at + n + 2 * y + 1] = hi;
            }
            at += n;
        }
    }
    const E2* weights(size_t half) const { return w_.data() + (half - 1); }
    // ---- host tables ----
    E2 total(int k) {   // before any fold: sum over the whole cube
        const E2 *a = ta_.data() + k * tn_, *b = tb_.data() + k * tn_;
        typename H::Dot d;
        const bool has = !pt_.empty();
        const E2* w = weights(tn_ / 2);
        for (size_t y = 0; 2 * y < tn_; y++) {
            E2 x0 = H::mul(a[2 * y], b[2 * y]), x1 = H::mul(a[2 * y + 1], b[2 * y + 1]);
            const E2 v = has ? H::add(x0, H::mul(pt_[0], H::sub(x1, x0))) : H::add(x0, x1);
            d.mac(w[y], v);
        }
        return d.value();
    }
    void host_sums(E2& s0, E2& s1, E2& s2) {
        const size_t half = live_ / 2;
        const bool weigh = (int)pt_.size() > round_ + 1;
        if (weigh && !have_w_) suffix(round_, n_);
        have_w_ = true;
        if (words_ && !weigh && scale_.empty()) {   // base field words still: one product instead of four
            typename H::Wide p0, p1, p2;
            for (size_t y = 0; y < half; y++) {
                const uint64_t a0 = ta_[2 * y].c0, a1 = ta_[2 * y + 1].c0, b0 = tb_[2 * y].c0, b1 = tb_[2 * y + 1].c0;
                p0.mac(a0, b0);
                p1.mac(a1, b1);
                p2.mac(O::sub(a1, a0), O::sub(b1, b0));
            }
            s0 = E2{O::canon(p0.red()), 0}; s1 = E2{O::canon(p1.red()), 0}; s2 = E2{O::canon(p2.red()), 0};
            return;
        }
        typename H::Dot d0, d1, d2;
        for (int k = 0; k < K_; k++) {
            const E2 *a = ta_.data() + k * tn_, *b = tb_.data() + k * tn_;
            typename H::Dot e0, e1, e2;
            typename H::Dot &f0 = scale_.empty() ? d0 : e0, &f1 = scale_.empty() ? d1 : e1, &f2 = scale_.empty() ? d2 : e2;
            for (size_t y = 0; y < half; y++) {
                E2 a0 = a[2 * y], a1 = a[2 * y + 1];
                if (weigh) {
                    const E2 w = weights(half)[y];
                    a0 = H::mul(w, a0);
                    a1 = H::mul(w, a1);
                }
                f0.mac(a0, b[2 * y]);
                f1.mac(a1, b[2 * y + 1]);
                f2.mac(H::sub(a1, a0), H::sub(b[2 * y + 1], b[2 * y]));
            }
            if (!scale_.empty()) {
                d0.mac(scale_[k], e0.value());
                d1.mac(scale_[k], e1.value());
                d2.mac(scale_[k], e2.value());
            }
        }
        s0 = d0.value(); s1 = d1.value(); s2 = d2.value();
    }
    void host_fold(E2 r) {
        const size_t half = live_ / 2;
        for (int k = 0; k < K_; k++)
            for (E2* t : {ta_.data() + k * tn_, tb_.data() + k * tn_})
                for (size_t y = 0; y < half; y++) {
                    if (words_) {
                        const uint64_t x = t[2 * y].c0, d = O::sub(t[2 * y + 1].c0, x);
                        t[y] = E2{O::canon(O::red((hf::u128)r.c0 * d + x)), O::canon(O::red((hf::u128)r.c1 * d))};
                    } else {
                        t[y] = H::fold(t[2 * y], t[2 * y + 1], r);
                    }
                }
        words_ = false;
        live_ = half;
    }

    const uint64_t *a_ = nullptr, *b_ = nullptr;
    size_t stride_ = 0, arriving_ = 0;   // words of pin_ that the pass queued last writes
    int K_ = 1, n_ = 0, cap_ = 1, round_ = 0, tail_first_ = 0, bad_ = MB_OK;
    bool base_ = false, flip_ = false, pending_ = false, host_ = false, weighted_ = false, have_w_ = false, words_ = false;
    std::vector<Block> blocks_;
    size_t block_ = 0;
    std::vector<E2> pt_, r_, scale_, m_, w_, ta_, tb_;
    int side_ = 0, width_ = 0;
    size_t tn_ = 0, live_ = 0;
    E2 eq_scale_{1, 0};
    ScratchBlock scratch_;
    uint64_t *pin_ = nullptr, *t0_ = nullptr, *t1_ = nullptr, *tabs_ = nullptr;
};

}  // namespace mbhost
