// Host side of the several-rounds-per-pass sumcheck over products of one table, three, or four small ones
// (product_kernels.cuh, product_mma_kernels.cuh). The object plans the blocks of rounds, queues the passes, runs the rounds of a block on the
// sums they return, and hands over the folded tables once they are small enough for the host.
//
//   rounds per block   one table: 4. Three tables: 3 up to 2^14 elements, then 2, on the tensor cores
//                      (product_mma_kernels.cuh). Four tables: 2. Each is where the pass's products cost about what the
//                      launch and the synchronisation of a round more do.
//   limit(d)           the largest tables (log2) this is for: with four tables two rounds at 2^14 take as long as two
//                      launches more; one table has no products, three have them on the tensor cores.
//   host tables        at most 2^8 elements, 2^7 where a pass can end there: the rest of a proof on them takes a core 10 to 20 us.
#pragma once
#include <vector>
#include "../product_kernels.cuh"
#include "../product_mma_kernels.cuh"
#include "pair_sumcheck.cuh"

namespace mbhost {

using namespace mb;

template <class F, class O>
class ProductSumcheck {
public:
    using H = PairHost<F, O>;
    using E2 = typename F::E2;
    static bool handles(int d) { return d == 1 || d == 3 || d == 4; }
    static int limit(int d) { return d == 4 ? 13 : 40; }
    ~ProductSumcheck() {
        if (scratch_) {   // nothing may still be writing it
            const bool clean = cudaStreamSynchronize(MB_STREAM) == cudaSuccess;
            ScratchPool::give(scratch_, clean && bad_ == MB_OK && pin_[ERROR_WORD] == 0);
        }
        pool_free(t0_);
        pool_free(t1_);
    }
    // d device tables of 2^vars elements, `stride` words apart (never written); r: a challenge they have still to be
    // folded on (four tables that were too large before it), or null. Queues the first pass.
    int init(const uint64_t* in, size_t stride, int d, int vars, bool base, const E2* r) {
        in_ = in; stride_ = stride; d_ = d; n_ = vars; base_ = base;
        r_.resize(vars);
        if (r) {
            r_[0] = *r;
            blocks_.push_back(Block{0, 1, false});
            block_ = 1;
            round_ = 1;
        }
        int v = vars - round_;
        while (v > 8) {
            int g = d == 1 ? 4 : d == 3 && v <= 14 ? 3 : 2;
            if (g > v - (d == 1 ? 8 : 7)) g = v - (d == 1 ? 8 : 7);
            blocks_.push_back(Block{n_ - v, g, d == 3 && v > MMA_ABOVE});
            v -= g;
        }
        tail_vars_ = v;
        scratch_ = ScratchPool::take();
        if (!scratch_) return MB_ERR_CUDA;
        pin_ = scratch_.host;
        pin_[ERROR_WORD] = 0;
        return failed(pass());
    }
    // Every round that is left is the host's: tables() has them.
    bool at_tail() const { return block_ == blocks_.size(); }
    // [d][2^tail] elements, canonical
    int tables(std::vector<E2>& tab, size_t& stride) {
        int rc = wait();
        if (rc != MB_OK) return rc;
        stride = (size_t)1 << tail_vars_;
        tab.resize(d_ * stride);
        const int nw = base_ ? 1 : 2;
        for (size_t j = 0; j < tab.size(); j++) tab[j] = H::canon(E2{pin_[nw * j], nw == 2 ? pin_[nw * j + 1] : 0});
        return MB_OK;
    }
    // P(0..d) of the current round
    int message(E2* p) {
        int rc = load();
        if (rc != MB_OK) return rc;
        E2 k[5];   // k[w]: sum of the entries whose low bits have w ones and whose other bits agree
        for (int w = 0; w <= d_; w++) k[w] = E2{0, 0};
        const int half = side_ / 2;
        for (int m = 0; m < half; m++)
            for (int b = 0; b < (1 << d_); b++) {
                size_t at = 0;
                int w = 0;
                for (int j = 0; j < d_; j++) {
                    const int bit = (b >> j) & 1;
                    at = at * side_ + 2 * m + bit;
                    w += bit;
                }
                k[w] = H::add(k[w], t_[at]);
            }
        for (int c = 0; c <= d_; c++) {   // sum_w k[w] c^w (1 - c)^(d - w)
            p[c] = E2{0, 0};
            for (int w = 0; w <= d_; w++) {
                uint64_t f = 1;
                for (int j = 0; j < w; j++) f *= c;
                for (int j = 0; j < d_ - w; j++) f *= c > 0 ? c - 1 : 1;
                const E2 x{O::canon(O::red((hf::u128)k[w].c0 * f)), O::canon(O::red((hf::u128)k[w].c1 * f))};
                p[c] = c > 1 && ((d_ - w) & 1) ? H::sub(p[c], x) : H::add(p[c], x);
            }
            p[c] = H::canon(p[c]);
        }
        return MB_OK;
    }
    int fold(E2 r) {
        int rc = load();
        if (rc != MB_OK) return rc;
        const int round = round_++;
        r_[round] = r;
        const Block& bl = blocks_[block_];
        if (round + 1 == bl.first + bl.rounds) {
            block_++;
            return failed(pass());
        }
        // one axis after the other: the last one is halved and moved to the front
        const int half = side_ / 2;
        size_t rows = t_.size() / side_;
        std::vector<E2> u(t_.size() / 2);
        for (int axis = 0; axis < d_; axis++) {
            for (size_t i = 0; i < rows; i++)
                for (int j = 0; j < half; j++) u[j * rows + i] = H::fold(t_[i * side_ + 2 * j], t_[i * side_ + 2 * j + 1], r);
            t_.assign(u.begin(), u.begin() + rows * half);
            rows = t_.size() / (axis + 1 < d_ ? side_ : half);
        }
        side_ = half;
        return MB_OK;
    }

private:
    static constexpr size_t ERROR_WORD = ScratchPool::WORDS - 2;
    static constexpr int MMA_ABOVE = 14;
    struct Block {
        int first, rounds;
        bool mma;   // three tables, two rounds: tri_mma_kernel
    };
    int pass() {
        const int from = block_ > 0 ? blocks_[block_ - 1].first : 0, fb = block_ > 0 ? blocks_[block_ - 1].rounds : 0;
        const bool last = at_tail();
        pr::FoldWeights<F> fw;
        E2 e[1 << pr::MAX_B];
        H::eq_vector(r_.data() + from, fb, e);
        for (int i = 0; i < (1 << fb); i++)
            fw.w[i] = typename F::Pre{H::canon(e[i]).c0, H::canon(e[i]).c1, O::canon(O::red((hf::u128)e[i].c1 * O::W))};
        pr::ProductArgs p{};
        p.fb = fb;
        p.in = in_; p.stride = stride_;
        p.v = n_ - (last ? n_ - tail_vars_ : blocks_[block_].first);
        p.acc = scratch_.dev; p.sums = pin_;
        loaded_ = false;
        arriving_ = 0;
        if (last) {
            p.out = pin_;
            if (fb == 0) return copy(p.v);
        } else if (fb) {
            uint64_t*& t = flip_ ? t1_ : t0_;
            if (!t) MB_CUDA(pool_alloc((void**)&t, sizeof(uint64_t) * ((size_t)2 << p.v) * d_));
            p.out = t;
            flip_ = !flip_;
        }
        arriving_ = 2 * (last ? (size_t)d_ << p.v : blocks_[block_].mma ? (size_t)pr::TRI_ENTRIES : (size_t)1 << (blocks_[block_].rounds * d_));
        expect_words(pin_, arriving_);
        if (!last && blocks_[block_].mma) {
            int rc = launch_mma(p, fw);
            if (rc != MB_OK) return rc;
        } else {
            const int gb = last ? 0 : blocks_[block_].rounds;
            MB_KERNEL(d_ == 1 ? "product_pass" : "product_tile");
            if (d_ == 1) launch_one(gb, fb > 0, p, fw);
            else if (d_ == 3) launch_three(gb, fb > 0, p, fw);
            else launch_four(gb, fb > 0, p, fw);
        }
        if (fb) {
            base_ = false;
            if (!last) {
                in_ = p.out;
                stride_ = (size_t)2 << p.v;
            }
        }
        return finish_async();
    }
    template <bool FOLD, bool BASE>
    static int launch_mma_as(unsigned grid, const pr::TriArgs& p, const pr::FoldWeights<F>& fw) {
        constexpr uint32_t smem = FOLD ? pr::TRI_FOLD_SMEM : pr::TRI_RAW_SMEM;
        const auto k = pr::tri_mma_kernel<F, FOLD, BASE>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return MB_ERR_CUDA;
        k<<<grid, pr::TRI_BLK, smem, MB_STREAM>>>(p, fw);
        return MB_OK;
    }
    int launch_mma(const pr::ProductArgs& q, const pr::FoldWeights<F>& fw) const {
        pr::TriArgs p{};
        p.in = q.in; p.stride = q.stride; p.out = q.out; p.v = q.v;
        p.acc = q.acc; p.sums = q.sums; p.error = pin_ + ERROR_WORD;
        const size_t tiles = ((size_t)1 << q.v) / (4 * pr::TRI_Y), least = (tiles + pr::TRI_MOST - 1) / pr::TRI_MOST;
        const size_t sms = (size_t)sm_count() > least ? (size_t)sm_count() : least;
        const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
        MB_KERNEL("product_mma");
        if (q.fb) return base_ ? launch_mma_as<true, true>(grid, p, fw) : launch_mma_as<true, false>(grid, p, fw);
        return base_ ? launch_mma_as<false, true>(grid, p, fw) : launch_mma_as<false, false>(grid, p, fw);
    }
    template <int GB>
    void launch_one(bool fold, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        const size_t tiles = ((size_t)1 << p.v) / pr::BLK, most = GB > 0 ? 8 * (size_t)sm_count() : tiles;
        const unsigned grid = tiles == 0 ? 1u : (unsigned)(tiles < most ? tiles : most);
        if (fold) {
            if (base_) pr::product_pass_kernel<F, GB, true, true><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
            else pr::product_pass_kernel<F, GB, true, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
        } else if constexpr (GB > 0) {
            if (base_) pr::product_pass_kernel<F, GB, false, true><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
            else pr::product_pass_kernel<F, GB, false, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
        }
    }
    void launch_one(int gb, bool fold, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        switch (gb) {
            case 0: launch_one<0>(fold, p, fw); break;
            case 1: launch_one<1>(fold, p, fw); break;
            case 2: launch_one<2>(fold, p, fw); break;
            case 3: launch_one<3>(fold, p, fw); break;
            default: launch_one<4>(fold, p, fw); break;
        }
    }
    template <int D, int GB, int PT>
    void launch_tiles(bool fold, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        // with sums 2^9 elements or more, at least four clusters; else the host's tables, 2^7 or 2^8
        static_assert(512 / PT % pr::PRODUCT_CLUSTER == 0 && 128 % PT == 0, "whole clusters, whole tiles");
        const unsigned grid = (unsigned)(((size_t)1 << p.v) / PT);
        const int s = !fold || PT > 16 ? 0 : p.fb > 2 ? 2 : p.fb - 1;   // a thread folds two inputs or more
        if (fold) {
            if (base_) pr::product_tile_kernel<F, D, GB, true, true, PT><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
            else pr::product_tile_kernel<F, D, GB, true, false, PT><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
        } else if constexpr (GB > 0) {
            if (base_) pr::product_tile_kernel<F, D, GB, false, true, PT><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
            else pr::product_tile_kernel<F, D, GB, false, false, PT><<<grid, pr::BLK, 0, MB_STREAM>>>(p, s, fw);
        }
    }
    // Tiles of 16 elements for three tables of up to 2^13 elements, of 64 for 2^14: a whole proof at 2^13 takes 99 or 101 us, at 2^14 117 or
    // 113 (four blocks an SM of the smaller ones wait for one another's sums). Four tables have at most 2^13: 123 or 127 us there.
    static constexpr int SMALL_TILES_TO = 13;
    void launch_three(int gb, bool fold, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {   // two rounds: of 2^9 elements
        if (gb == 0) launch_tiles<3, 0, 16>(fold, p, fw);
        else if (gb == 2) launch_tiles<3, 2, 16>(fold, p, fw);
        else if (p.v <= SMALL_TILES_TO) launch_tiles<3, 3, 16>(fold, p, fw);
        else launch_tiles<3, 3, 64>(fold, p, fw);
    }
    void launch_four(int gb, bool fold, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        if (gb == 0) launch_tiles<4, 0, 16>(fold, p, fw);
        else launch_tiles<4, 2, 16>(fold, p, fw);
    }
    // tables that no pass has folded come as they are
    int copy(int v) {
        const size_t w = ((size_t)1 << v) * (base_ ? 1 : 2);
        arriving_ = w * d_;
        expect_words(pin_, arriving_);
        MB_KERNEL("product_tables");
        pr::send_tables_kernel<F><<<dim3((unsigned)((w + pr::BLK - 1) / pr::BLK), d_), pr::BLK, 0, MB_STREAM>>>(in_, in_ + stride_, 2 * stride_, w, pin_);
        return finish_async();
    }
    // As PairSumcheck: after a failure every later call fails.
    int failed(int rc) {
        if (rc != MB_OK) bad_ = rc;
        return rc;
    }
    int wait() {
        if (bad_ != MB_OK) return bad_;
        if (await_words(pin_, arriving_) != MB_OK) return failed(MB_ERR_CUDA);
        return failed(pin_[ERROR_WORD] != 0 ? MB_ERR_CUDA : MB_OK);
    }
    // The sums of the current block.
    int load() {
        if (bad_ == MB_OK && loaded_) return MB_OK;
        int rc = wait();
        if (rc != MB_OK) return rc;
        const int g = blocks_[block_].rounds;
        side_ = 1 << g;
        t_.resize((size_t)1 << (g * d_));
        if (blocks_[block_].mma) expand();
        else for (size_t j = 0; j < t_.size(); j++) t_[j] = E2{pin_[2 * j], pin_[2 * j + 1]};
        loaded_ = true;
        return MB_OK;
    }

    // The rounds only use f g as a polynomial: with its values q0, q1 and leading coefficient q2 in a variable, entries
    // (0, 0) = q0, (1, 1) = q1, (0, 1) = q0 + q1 - q2 and (1, 0) = 0 of the two tables give the same one.
    void expand() {
        const auto q = [&](int p, int k) { return E2{pin_[2 * (4 * p + k)], pin_[2 * (4 * p + k) + 1]}; };
        for (int i = 0; i < 4; i++)
            for (int j = 0; j < 4; j++)
                for (int k = 0; k < 4; k++) {
                    const int first = 2 * (i & 1) + (j & 1), second = 2 * (i >> 1) + (j >> 1);   // of table f and g, in each variable
                    const auto in_first = [&](int p1) {
                        if (first == 0) return q(3 * p1, k);
                        if (first == 3) return q(3 * p1 + 1, k);
                        return H::sub(H::add(q(3 * p1, k), q(3 * p1 + 1, k)), q(3 * p1 + 2, k));
                    };
                    E2& t = t_[(4 * i + j) * 4 + k];
                    if (first == 2 || second == 2) t = E2{0, 0};
                    else if (second == 0) t = in_first(0);
                    else if (second == 3) t = in_first(1);
                    else t = H::sub(H::add(in_first(0), in_first(1)), in_first(2));
                }
    }

    const uint64_t* in_ = nullptr;
    size_t stride_ = 0, arriving_ = 0;   // as in PairSumcheck
    int d_ = 0, n_ = 0, round_ = 0, side_ = 0, tail_vars_ = 0, bad_ = MB_OK;
    bool base_ = false, flip_ = false, loaded_ = false;
    std::vector<Block> blocks_;
    size_t block_ = 0;
    std::vector<E2> r_, t_;
    ScratchBlock scratch_;
    uint64_t *pin_ = nullptr, *t0_ = nullptr, *t1_ = nullptr;
};

}  // namespace mbhost
