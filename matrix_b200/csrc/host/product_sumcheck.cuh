// Host side of the several-rounds-per-pass sumcheck over products of one, three or four small tables
// (product_kernels.cuh). The object plans the blocks of rounds, queues the passes, runs the rounds of a block on the
// sums they return, and hands over the folded tables once they are small enough for the host.
//
//   rounds per block   one table: 4. Three tables: 3 up to 2^14 elements, then 2. Four tables: 2. Each is where the
//                      pass's products cost about what the launch and the synchronisation of a round more do.
//   limit(d)           the largest tables (log2) this is for: with three tables two rounds at 2^17 take 15 us of
//                      products against two launches; with four tables the same holds at 2^14; one table has no products.
//   host tables        at most 2^8 elements, 2^7 where a pass can end there: the rest of a proof on them takes a core 10 to 20 us.
#pragma once
#include <vector>
#include "../product_kernels.cuh"
#include "pair_sumcheck.cuh"

namespace mbhost {

using namespace mb;

template <class F, class O>
class ProductSumcheck {
public:
    using H = PairHost<F, O>;
    using E2 = typename F::E2;
    static bool handles(int d) { return d == 1 || d == 3 || d == 4; }
    static int limit(int d) { return d == 1 ? 40 : d == 3 ? 16 : 13; }
    ~ProductSumcheck() {
        if (scratch_) ScratchPool::give(scratch_, cudaStreamSynchronize(MB_STREAM) == cudaSuccess);   // nothing may still be writing it
        pool_free(t0_);
        pool_free(t1_);
    }
    // d device tables of 2^vars elements, `stride` words apart (never written); r: a challenge they have still to be
    // folded on, or null. Queues the first pass.
    int init(const uint64_t* in, size_t stride, int d, int vars, bool base, const E2* r) {
        in_ = in; stride_ = stride; d_ = d; n_ = vars; base_ = base;
        r_.resize(vars);
        if (r) {
            r_[0] = *r;
            blocks_.push_back(Block{0, 1});
            block_ = 1;
            round_ = 1;
        }
        int v = vars - round_;
        while (v > 8) {
            int g = d == 1 ? 4 : d == 3 && v <= 14 ? 3 : 2;
            if (g > v - (d == 1 ? 8 : 7)) g = v - (d == 1 ? 8 : 7);
            blocks_.push_back(Block{n_ - v, g});
            v -= g;
        }
        tail_vars_ = v;
        scratch_ = ScratchPool::take();
        if (!scratch_) return MB_ERR_CUDA;
        pin_ = scratch_.host;
        cap_ = sm_count() * (d == 1 ? 8 : 4);
        return pass();
    }
    // Every round that is left is the host's: tables() has them.
    bool at_tail() const { return block_ == blocks_.size(); }
    // [d][2^tail] elements, canonical
    int tables(std::vector<E2>& tab, size_t& stride) {
        MB_CUDA(cudaStreamSynchronize(MB_STREAM));
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
            return pass();
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
    struct Block { int first, rounds; };
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
        if (last) {
            p.out = pin_;
            if (fb == 0) return copy(p.v);
        } else if (fb) {
            uint64_t*& t = flip_ ? t1_ : t0_;
            if (!t) MB_CUDA(pool_alloc((void**)&t, sizeof(uint64_t) * ((size_t)2 << p.v) * d_));
            p.out = t;
            flip_ = !flip_;
        }
        const size_t tiles = ((size_t)1 << p.v) / (d_ == 1 ? pr::BLK : pr::PTILE);
        const unsigned grid = last ? (tiles ? (unsigned)tiles : 1u) : tiles < (size_t)cap_ ? (unsigned)tiles : (unsigned)cap_;
        const int gb = last ? 0 : blocks_[block_].rounds;
        {
            MB_KERNEL("product_pass");
            if (d_ == 1) launch_d<1>(gb, fb > 0, grid, p, fw);
            else if (d_ == 3) launch_d<3>(gb, fb > 0, grid, p, fw);
            else launch_d<4>(gb, fb > 0, grid, p, fw);
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
    template <int D, int GB>
    void launch(bool fold, unsigned grid, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        if (fold) {
            if (base_) pr::product_pass_kernel<F, D, GB, true, true><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
            else pr::product_pass_kernel<F, D, GB, true, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
        } else if constexpr (GB > 0) {
            if (base_) pr::product_pass_kernel<F, D, GB, false, true><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
            else pr::product_pass_kernel<F, D, GB, false, false><<<grid, pr::BLK, 0, MB_STREAM>>>(p, fw);
        }
    }
    template <int D>
    void launch_d(int gb, bool fold, unsigned grid, const pr::ProductArgs& p, const pr::FoldWeights<F>& fw) const {
        switch (gb) {
            case 0: launch<D, 0>(fold, grid, p, fw); break;
            case 1: launch<D, 1>(fold, grid, p, fw); break;
            case 2: launch<D, 2>(fold, grid, p, fw); break;
            case 3: if constexpr (D != 4) launch<D, 3>(fold, grid, p, fw); break;
            default: if constexpr (D == 1) launch<D, 4>(fold, grid, p, fw); break;
        }
    }
    // tables that no pass has folded come as they are
    int copy(int v) {
        const size_t w = ((size_t)1 << v) * (base_ ? 1 : 2);
        for (int k = 0; k < d_; k++)
            MB_CUDA(cudaMemcpyAsync(pin_ + w * k, in_ + stride_ * k, 8 * w, cudaMemcpyDeviceToHost, MB_STREAM));
        return MB_OK;
    }
    // The sums of the current block.
    int load() {
        if (loaded_) return MB_OK;
        MB_CUDA(cudaStreamSynchronize(MB_STREAM));
        const int g = blocks_[block_].rounds;
        side_ = 1 << g;
        t_.resize((size_t)1 << (g * d_));
        for (size_t j = 0; j < t_.size(); j++) t_[j] = E2{pin_[2 * j], pin_[2 * j + 1]};
        loaded_ = true;
        return MB_OK;
    }

    const uint64_t* in_ = nullptr;
    size_t stride_ = 0;
    int d_ = 0, n_ = 0, cap_ = 1, round_ = 0, side_ = 0, tail_vars_ = 0;
    bool base_ = false, flip_ = false, loaded_ = false;
    std::vector<Block> blocks_;
    size_t block_ = 0;
    std::vector<E2> r_, t_;
    ScratchBlock scratch_;
    uint64_t *pin_ = nullptr, *t0_ = nullptr, *t1_ = nullptr;
};

}  // namespace mbhost
