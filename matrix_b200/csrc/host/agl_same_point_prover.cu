// Same-point sumcheck over the almost-Goldilocks extension, whole protocol: the host loop the reference keeps
// in Rust (zk-torch-4/src/fold/same_point_sumcheck.rs), over this library's batched same-point kernels.
//
//   prove_same_point_gpu_batched           same_point_sumcheck.rs:1032-1063, 1334-1553 (uniform arity: header,
//                                          alpha, device eq tables, per-round combined message, fold, reveals)
//   GpuBatchedSamePointState               almost-goldilocks-cuda-rs/src/sumcheck_prover.rs:468-760 (interleaved
//                                          layout: per leaf the eq table, then the f table)
//   verify_same_point                      same_point_sumcheck.rs:161-219
//
// M instances of the same arity k, each with its own claim point r_i, claim y_i = f_i(r_i) and witness f_i
// (binary packed, ternary single chunk, or an extension table); the sumcheck
//   sum_i alpha^i y_i = sum_x sum_i alpha^i eq(r_i, x) f_i(x)
// reduces them to one point R. Degree 2: three evaluations per round. The transcript is the caller's (Monolith
// width 12) and is advanced exactly as the reference's prover advances it, so proofs are interchangeable with
// the CPU prover's (heterogeneous arities stay on that path, as in the reference).
//
// Device side (same_point_kernels.cuh): the eq polynomials stay factored, and one pass over a table serves up to four
// rounds (six for the packed witness): it returns the 3^B values of the rounds' polynomial over all leaves, or 2^B eq-weighted
// sums per leaf where there are few, on which the host runs the messages and folds of B rounds, and the next pass folds the B
// challenges at once. The first pass is queued before the header of
// the transcript (every claim point, label by label), which the host absorbs while the device works: after the pass
// that header is the longest part of a proof. The reference launches a message and a fold kernel per round over eq and f
// tables; with one fused pass per round over both tables, arity 22 and 42 binary leaves took 7.4 ms and 11 GB.
#include <vector>
#include "../same_point_kernels.cuh"
#include "agl_transcript.hpp"
#include "arrivals.hpp"
#include "host_field.hpp"
#include "scratch_pool.hpp"

using namespace mb;
using namespace mb::sc;

namespace mbhost {

using AglTranscript = aglm::Transcript;
using E2 = agl::E2;

namespace {

const uint8_t L_NUM_VAR[] = "sp_num_var", L_NUM_INST[] = "sp_num_inst", L_ARITY[] = "sp_arity_i", L_R[] = "sp_r_i",
              L_Y[] = "sp_y_i", L_ALPHA[] = "sp_alpha", L_MSG[] = "sp_round_msg", L_CH[] = "sp_round_challenge",
              L_FEVAL[] = "sp_f_eval";
#define SP_LABEL(l) l, sizeof(l) - 1

inline E2 e2c(E2 a) { return agl::e2_canon(a); }
inline E2 ld(const uint64_t* w) { return E2{agl::canon(w[0]), agl::canon(w[1])}; }
inline E2 challenge(AglTranscript& t, const uint8_t* l, size_t n) {
    uint64_t w[2];
    t.challenge_vector(l, n, w, 2);   // the label once, two squeezes (transcript.rs:120-125)
    return E2{w[0], w[1]};
}

void header(AglTranscript& t, int M, int arity, const uint64_t* pts, const uint64_t* vals) {   // same_point_sumcheck.rs:78-87
    t.append_u64(SP_LABEL(L_NUM_VAR), (uint64_t)arity);
    t.append_u64(SP_LABEL(L_NUM_INST), (uint64_t)M);
    for (int i = 0; i < M; i++) {
        t.append_u64(SP_LABEL(L_ARITY), (uint64_t)arity);
        for (int k = 0; k < arity; k++) {
            const uint64_t* p = pts + ((size_t)i * arity + k) * 2;
            t.append_ext2(SP_LABEL(L_R), p[0], p[1]);
        }
        t.append_ext2(SP_LABEL(L_Y), vals[2 * i], vals[2 * i + 1]);
    }
}

E2 eq_eval(const uint64_t* a, const E2* b, int n) {   // same_point_sumcheck.rs:907-921
    E2 acc{1, 0};
    const E2 one{1, 0};
    for (int i = 0; i < n; i++) {
        const E2 ai = ld(a + 2 * i);
        acc = e2c(agl::e2_mul(acc, agl::e2_add(agl::e2_mul(ai, b[i]), agl::e2_mul(agl::e2_sub(one, ai), agl::e2_sub(one, b[i])))));
    }
    return acc;
}

// ---- the rounds of one pass on the host -------------------------------------------------------
E2 mul(E2 a, E2 b) {   // canonical words in and out, on the host core's multiplier
    E2 r;
    hf::e2_mul<hf::AglE2Ops>(a.c0, a.c1, b.c0, b.c1, r.c0, r.c1);
    return r;
}
E2 add(E2 a, E2 b) { return E2{hf::agl_add(a.c0, b.c0), hf::agl_add(a.c1, b.c1)}; }
E2 sub(E2 a, E2 b) { return E2{hf::agl_sub(a.c0, b.c0), hf::agl_sub(a.c1, b.c1)}; }
// sum of products, reduced once
struct Dot {
    struct Wide {
        hf::u128 s = 0;
        uint64_t top = 0;
        void mac(uint64_t x, uint64_t y) {
            const hf::u128 p = (hf::u128)x * y;
            s += p;
            top += s < p;
        }
        // 2^128 = 63 2^32 + 992 (mod q)
        uint64_t red() const { return hf::agl_red((hf::u128)top * (63ULL * (1ULL << 32) + 992ULL) + hf::agl_red(s)); }
    };
    Wide p00, p11, p01;
    void mac(E2 a, E2 b) {
        p00.mac(a.c0, b.c0);
        p11.mac(a.c1, b.c1);
        p01.mac(a.c0, b.c1);
        p01.mac(a.c1, b.c0);
    }
    E2 value() const {
        return E2{hf::agl_canon(hf::agl_red((hf::u128)p11.red() * 3 + p00.red())), hf::agl_canon(p01.red())};
    }
};

// A block of rounds from variable `first` on, and what the pass before it reads.
enum Source { FROM_WITNESS, FROM_WORD_SUMS, FROM_WORDS, FROM_TABLE };
struct Stage {
    int first, rounds;
    Source source;
    size_t wl = 0, wh = 0;
};

struct Buffers {
    uint64_t *pts = nullptr, *tabs = nullptr, *partial = nullptr, *g6 = nullptr, *t0 = nullptr, *t1 = nullptr, *scale = nullptr;
    unsigned* counter = nullptr;
    ~Buffers() {
        pool_free(pts); pool_free(scale); pool_free(tabs); pool_free(partial); pool_free(g6); pool_free(t0); pool_free(t1); pool_free(counter);
    }
};

// Page-locked landing zone of the calling thread for the sums (grown on demand, kept between calls): the last block of
// a pass writes them there.
uint64_t* pinned_words(size_t words) {
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

class SamePointDevice {
public:
    ~SamePointDevice() {
        if (scratch_) ScratchPool::give(scratch_, cudaStreamSynchronize(MB_STREAM) == cudaSuccess);
    }
    // Stages of the proof, eq tables of all passes, and the first pass, all queued; the sums of the first stage are in
    // sums() after wait(). claims_only: nothing after the first pass will be asked for; share: later stages
    // return the values of their rounds' polynomial, else each leaf's sums.
    int init(int M, int arity, const uint64_t* h_pts, int kind, const uint64_t* d_w0, const uint64_t* d_w1, bool claims_only, bool share) {
        M_ = M; share_ = share; k_ = arity; kind_ = kind; w0_ = d_w0; w1_ = d_w1;
        const int inside = kind == 2 ? 0 : (arity < sp::BITS ? arity : sp::BITS);
        words_ = arity >= 6 ? (size_t)1 << (arity - 6) : 1;
        if (inside) {
            const int b0 = (inside + 1) / 2;
            stages_.push_back({0, b0, FROM_WITNESS});
            if (inside > b0) stages_.push_back({b0, inside - b0, FROM_WORD_SUMS});
        }
        const int rest = arity - inside, parts = (rest + sp::MAX_B - 1) / sp::MAX_B;
        for (int i = 0, at = inside; i < parts; i++) {
            const int b = (arity - at + (parts - i) - 1) / (parts - i);
            stages_.push_back({at, b, at == inside ? (inside ? FROM_WORDS : FROM_WITNESS) : FROM_TABLE});
            at += b;
        }
        // eq tables: per pass over the variables the thread index and the loop counter stand for
        sp::TableSet set;
        int nt = 0;
        const auto table = [&](int first, int bits) {
            set.d[nt].first = first;
            set.d[nt].bits = bits;
            set.d[nt].off = leaf_words_;
            leaf_words_ += (size_t)4 << bits;
            return set.d[nt++].off;
        };
        size_t low_off = 0;
        const int lo_bits = rest < 8 ? rest : 8;
        for (Stage& s : stages_) {
            if (s.source == FROM_WITNESS && inside) {
                s.wl = table(inside, lo_bits);
                s.wh = table(inside + lo_bits, rest - lo_bits);
                low_off = table(s.rounds, inside - s.rounds);
            } else if (s.source != FROM_WORD_SUMS) {
                const int v = arity - s.first, tb = v < 8 ? v : 8;
                s.wl = table(s.first + s.rounds, tb - s.rounds);
                s.wh = table(s.first + tb, v - tb);
            }
            if (claims_only) break;
        }
        const int cap = sm_count() * 8 / M > 1 ? sm_count() * 8 / M : 1;
        max_blocks_ = cap;
        MB_CUDA(pool_alloc((void**)&b_.pts, sizeof(uint64_t) * 2 * (size_t)arity * M));
        MB_CUDA(pool_alloc((void**)&b_.tabs, sizeof(uint64_t) * leaf_words_ * M));
        MB_CUDA(pool_alloc((void**)&b_.partial, sizeof(uint64_t) * 2 * 64 * (size_t)cap * M));
        MB_CUDA(pool_alloc((void**)&b_.counter, sizeof(unsigned) * M));
        if (share_) {
            MB_CUDA(pool_alloc((void**)&b_.scale, sizeof(uint64_t) * 2 * (size_t)M));
            scratch_ = ScratchPool::take();
            if (!scratch_) return MB_ERR_CUDA;
        }
        if (inside) MB_CUDA(pool_alloc((void**)&b_.g6, sizeof(uint64_t) * 2 * 64 * (size_t)M));
        // staging: the points go up from page-locked memory, the sums come back behind them
        const size_t pt_words = 2 * (size_t)arity * M;
        uint64_t* pin = pinned_words(pt_words + ((size_t)2 << sp::MAX_B) * M);
        if (!pin) return MB_ERR_CUDA;
        for (size_t i = 0; i < pt_words; i++) pin[i] = h_pts[i];
        h_sums_ = pin + pt_words;
        MB_CUDA(cudaMemcpyAsync(b_.pts, pin, sizeof(uint64_t) * pt_words, cudaMemcpyHostToDevice, MB_STREAM));
        MB_CUDA(cudaMemsetAsync(b_.counter, 0, sizeof(unsigned) * M, MB_STREAM));
        {
            MB_KERNEL("same_point_eq_tables");
            sp::eq_tables_kernel<<<dim3(nt, M), sp::BLK, 0, MB_STREAM>>>(set, b_.pts, arity, b_.tabs, leaf_words_);
        }
        if (!inside) return fold(0, nullptr, 0);
        sp::BitsArgs a;
        a.pos = d_w0; a.neg = d_w1; a.words = words_;
        a.lo_bits = lo_bits; a.hi_bits = rest - lo_bits; a.in_bits = inside; a.first_bits = stages_[0].rounds;
        a.tabs = b_.tabs; a.leaf_words = leaf_words_; a.wl_off = stages_[0].wl; a.wh_off = stages_[0].wh; a.low_off = low_off;
        a.partial = b_.partial; a.g6 = b_.g6; a.counter = b_.counter; a.out = h_sums_;
        expect_sums(stages_[0]);
        // eight warps a block, a warp per high index: a power of two of blocks, so that no warp has more of them
        int gx = 1;
        while (2 * gx <= cap && (size_t)16 * gx <= ((size_t)1 << a.hi_bits)) gx *= 2;
        {
            MB_KERNEL("same_point_bits");
            if (kind == 1) sp::bits_pass_kernel<true><<<dim3(gx, M), sp::BLK, 0, MB_STREAM>>>(a);
            else sp::bits_pass_kernel<false><<<dim3(gx, M), sp::BLK, 0, MB_STREAM>>>(a);
        }
        return finish_async();
    }
    // The polynomial of the first stage's rounds, once alpha is known.
    int first_share(E2 alpha) {
        expect_values(stages_[0]);
        sums_words_ = 0;
        MB_KERNEL("same_point_share");
        sp::first_share_kernel<<<M_, sp::BLK, 0, MB_STREAM>>>(h_sums_, stages_[0].rounds, b_.pts, k_, alpha, b_.scale, scratch_.dev, scratch_.host);
        return finish_async();
    }
    // The pass before stage i: folds the challenges r[0 .. count) that bind the variables the pass consumes (all six of
    // a word for the first extension table, those of the stage before otherwise) and queues the sums of stage i.
    int fold(size_t i, const E2* r, int count) {
        const Stage& s = stages_[i];
        sp::FoldArgs a{};
        a.v = k_ - s.first;
        a.next = s.rounds;
        if (s.source == FROM_WORD_SUMS) a.v = s.rounds;   // the other variables are summed already
        a.t_bits = a.v < 8 ? a.v : 8;
        a.tabs = b_.tabs; a.leaf_words = leaf_words_; a.wl_off = s.wl; a.wh_off = s.wh;
        a.partial = b_.partial; a.counter = b_.counter;
        a.out = !share_ || i == 0 || i + 1 == stages_.size() ? h_sums_ : nullptr;   // for the first share; for the reveals
        if (a.out != nullptr) expect_sums(s);
        else sums_words_ = 0;
        if (share_ && i > 0) {
            expect_values(s);
            a.pts = b_.pts; a.arity = k_; a.first = s.first; a.bound = stages_[i - 1].rounds;
            a.scale = b_.scale; a.acc = scratch_.dev; a.u = scratch_.host;
            for (int j = 0; j < a.bound; j++) a.r[j] = r[count - a.bound + j];
        }
        const size_t iters = (size_t)1 << (a.v - a.t_bits);
        const int half = (max_blocks_ + 1) / 2, gx = iters < (size_t)half ? (int)iters : half;
        const dim3 grid(gx, M_);
        if (s.source == FROM_WORD_SUMS) {
            a.in = b_.g6; a.in_stride = 2 * 64;
        } else if (s.source == FROM_WORDS) {
            a.in = w0_; a.neg = w1_; a.in_stride = words_;
        } else {   // the caller's extension tables serve the first two passes
            a.in = kind_ == 2 && i <= 1 ? w0_ : cur_;
            a.in_stride = (size_t)2 << (a.v + count);
        }
        // a table is stored only for a pass that will read it
        if (i + 1 < stages_.size() && s.source != FROM_WITNESS && s.source != FROM_WORD_SUMS) {
            uint64_t*& t = flip_ ? b_.t1 : b_.t0;
            if (!t) MB_CUDA(pool_alloc((void**)&t, sizeof(uint64_t) * ((size_t)2 << a.v) * M_));
            a.table = cur_ = t;
            flip_ = !flip_;
        }
        if (s.source == FROM_WORDS) {
            sp::WordWeights w;
            eq_vector(r, count, w.w);
            for (int j = 1 << count; j < 64; j++) w.w[j] = E2{0, 0};
            MB_KERNEL("same_point_words");
            constexpr int lut = 8 * 256 * 16;
            if (kind_ == 1) launch<0, 2>(a.u != nullptr, grid, lut, a, w);
            else launch<0, 1>(a.u != nullptr, grid, lut, a, w);
            return finish_async();
        }
        sp::FoldWeights w;
        E2 e[1 << sp::MAX_B];
        eq_vector(r, count, e);
        for (int j = 0; j < (1 << count); j++) w.w[j] = agl::e2_pre(e[j]);
        MB_KERNEL("same_point_fold");
        switch (count) {
            case 0: launch<0, 0>(a.u != nullptr, grid, 0, a, w); break;
            case 1: launch<1, 0>(a.u != nullptr, grid, 0, a, w); break;
            case 2: launch<2, 0>(a.u != nullptr, grid, 0, a, w); break;
            case 3: launch<3, 0>(a.u != nullptr, grid, 0, a, w); break;
            default: launch<4, 0>(a.u != nullptr, grid, 0, a, w); break;
        }
        return finish_async();
    }
    // The results of the pass queued last.
    int wait() const {
        if (value_words_) {
            int rc = await_words(scratch_.host, value_words_);
            if (rc != MB_OK) return rc;
        }
        return await_words(h_sums_, sums_words_);
    }
    const std::vector<Stage>& stages() const { return stages_; }
    const uint64_t* sums() const { return h_sums_; }   // [leaf][2^rounds][2] of the stage queued last; share: of the first or the last
    const uint64_t* values() const { return scratch_.host; }   // [3^rounds][2] of the stage queued last

private:
    void expect_sums(const Stage& s) { expect_words(h_sums_, sums_words_ = ((size_t)2 << s.rounds) * M_); }
    void expect_values(const Stage& s) {
        value_words_ = 2;
        for (int j = 0; j < s.rounds; j++) value_words_ *= 3;
        expect_words(scratch_.host, value_words_);
    }
    template <int B, int SRC, class W>
    static void launch(bool share, dim3 grid, size_t smem, const sp::FoldArgs& a, const W& w) {
        if (share) sp::fold_pass_kernel<B, SRC, true, W><<<grid, sp::BLK, smem, MB_STREAM>>>(a, w);
        else sp::fold_pass_kernel<B, SRC, false, W><<<grid, sp::BLK, smem, MB_STREAM>>>(a, w);
    }
    // out[x] = prod_k (x_k ? r_k : 1 - r_k)
    static void eq_vector(const E2* r, int n, E2* out) {
        out[0] = E2{1, 0};
        for (int b = 0; b < n; b++)
            for (int x = 0; x < (1 << b); x++) {
                const E2 hi = mul(out[x], r[b]);
                out[x + (1 << b)] = hi;
                out[x] = sub(out[x], hi);
            }
    }
    int M_ = 0, k_ = 0, kind_ = 0, max_blocks_ = 1;
    size_t words_ = 1, leaf_words_ = 0, sums_words_ = 0, value_words_ = 0;   // the last two: of the pass queued last
    const uint64_t *w0_ = nullptr, *w1_ = nullptr;
    uint64_t *h_sums_ = nullptr, *cur_ = nullptr;
    bool flip_ = false, share_ = false;
    std::vector<Stage> stages_;
    ScratchBlock scratch_;
    Buffers b_;
};

}  // namespace

// y_i = f_i(r_i) for every leaf: the claims the protocol starts from (FoldData::evaluate_at_ext2,
// zk-torch-4/src/fold/mod.rs:107-110), as sum_m eq(r_i[0 .. B), m) G_i(m) over the sums of the first stage.
int same_point_claims(int M, int arity, const uint64_t* h_pts, int kind, const uint64_t* d_w0, const uint64_t* d_w1, uint64_t* h_vals) {
    if (M < 1 || M > 4096 || arity < 1 || arity > 32 || !h_pts || !d_w0 || kind < 0 || kind > 2 || (kind == 1 && !d_w1) || !h_vals)
        return MB_ERR_ARG;
    SamePointDevice dev;
    int rc = dev.init(M, arity, h_pts, kind, d_w0, d_w1, true, false);
    if (rc != MB_OK) return rc;
    rc = dev.wait();
    if (rc != MB_OK) return rc;
    const int b = dev.stages()[0].rounds;
    for (int i = 0; i < M; i++) {
        E2 g[1 << sp::MAX_B];
        for (int m = 0; m < (1 << b); m++) g[m] = ld(dev.sums() + 2 * (((size_t)i << b) + m));
        for (int j = 0; j < b; j++)
            for (int m = 0; m < (1 << (b - j - 1)); m++)
                g[m] = add(g[2 * m], mul(ld(h_pts + 2 * ((size_t)i * arity + j)), sub(g[2 * m + 1], g[2 * m])));
        h_vals[2 * i] = g[0].c0;
        h_vals[2 * i + 1] = g[0].c1;
    }
    return MB_OK;
}

// Leaves times rounds from which the shares are added up on the device: that takes 60 to 90 us a proof, the host's sums 0.2 us a
// leaf and round. By leaf / by share, us: 4 leaves of arity 8 99 / 136, 7 of arity 18 195 / 237, 30 of arity 12 267 / 284, 50 of
// arity 9 301 / 283, 30 of arity 21 497 / 430, 42 of arity 22 688 / 554.
constexpr int SHARE_FROM = 440;

namespace {
// The rounds on the 2^B sums of each leaf.
int rounds_by_leaf(SamePointDevice& dev, int M, int arity, const uint64_t* h_pts, E2 alpha, AglTranscript& t, uint64_t* h_round_msgs,
                   uint64_t* h_challenges, uint64_t* h_f_evals, uint64_t* h_final_eval) {
    // scale_i = alpha^i eq(r_i[0 .. j), R[0 .. j))
    std::vector<E2> scale(M);
    E2 pw{1, 0};
    for (int i = 0; i < M; i++) { scale[i] = pw; pw = mul(pw, alpha); }

    std::vector<E2> R(arity), g((size_t)M << sp::MAX_B), up(M), down(M);
    // suffix eq tables of the block's variables, per leaf: 2^(rounds - 1 - j) entries for round j, back to back
    std::vector<E2> suffix((size_t)M << sp::MAX_B);
    bool label_absorbed = false;
    for (size_t si = 0; si < dev.stages().size(); si++) {
        const Stage st = dev.stages()[si];
        if (si > 0) {
            // the challenges that the pass consumes: all of a word's for the first extension table
            const int from = st.source == FROM_WORDS ? 0 : dev.stages()[si - 1].first;
            int rc = dev.fold(si, R.data() + from, st.first - from);
            if (rc != MB_OK) return rc;
        }
        if (si > 0) {   // while the pass runs
            t.begin_append(SP_LABEL(L_MSG));
            label_absorbed = true;
        }
        const int B = st.rounds, size = 1 << B;
        for (int i = 0; i < M; i++) {
            // tables for rounds B - 1, B - 2, ..: each from the one before by its lowest variable
            E2* w = suffix.data() + ((size_t)i << B);
            w[0] = E2{1, 0};
            int at = 0;
            for (int j = B - 2; j >= 0; j--) {
                const E2 rj = ld(h_pts + 2 * ((size_t)i * arity + st.first + j + 1));
                const int n = 1 << (B - 2 - j);
                for (int y = 0; y < n; y++) {
                    const E2 hi = mul(w[at + y], rj);
                    w[at + n + 2 * y + 1] = hi;
                    w[at + n + 2 * y] = sub(w[at + y], hi);
                }
                at += n;
            }
        }
        int rc = dev.wait();
        if (rc != MB_OK) return rc;
        for (size_t x = 0; x < (size_t)M * size; x++) g[x] = E2{dev.sums()[2 * x], dev.sums()[2 * x + 1]};
        for (int j = 0; j < B; j++) {
            const int round = st.first + j, half = size >> (j + 1);
            // T_i(c) = scale_i ((1 - r)(1 - c) + r c) (A + c (B - A)) with A, B the weighted even and odd sums;
            // with u = scale (1 - r), v = scale r: T(0) = u A, T(1) = v B, T(2) = (2 v - u)(2 B - A)
            Dot m0, m1, m2;
            for (int i = 0; i < M; i++) {
                const E2* w = suffix.data() + ((size_t)i << B) + (half - 1);
                const E2* gi = g.data() + (size_t)i * size;
                E2 a = gi[0], b = gi[1];
                if (half > 1) {
                    Dot da, db;
                    for (int y = 0; y < half; y++) { da.mac(w[y], gi[2 * y]); db.mac(w[y], gi[2 * y + 1]); }
                    a = da.value();
                    b = db.value();
                }
                up[i] = mul(scale[i], ld(h_pts + 2 * ((size_t)i * arity + round)));
                down[i] = sub(scale[i], up[i]);
                m0.mac(down[i], a);
                m1.mac(up[i], b);
                m2.mac(sub(add(up[i], up[i]), down[i]), sub(add(b, b), a));
            }
            const E2 msg[3] = {m0.value(), m1.value(), m2.value()};
            for (int c = 0; c < 3; c++) {
                if (c > 0 || !label_absorbed) t.begin_append(SP_LABEL(L_MSG));
                t.finish_append_ext2(msg[c].c0, msg[c].c1);
                h_round_msgs[((size_t)round * 3 + c) * 2] = msg[c].c0;
                h_round_msgs[((size_t)round * 3 + c) * 2 + 1] = msg[c].c1;
            }
            label_absorbed = false;
            const E2 r = challenge(t, SP_LABEL(L_CH));
            R[round] = r;
            if (h_challenges) { h_challenges[2 * round] = r.c0; h_challenges[2 * round + 1] = r.c1; }
            const bool last = si + 1 == dev.stages().size();
            for (int i = 0; i < M; i++) {
                scale[i] = add(down[i], mul(r, sub(up[i], down[i])));
                if (j + 1 == B && !last) continue;   // the next pass folds
                E2* gi = g.data() + (size_t)i * size;
                for (int y = 0; y < half; y++) gi[y] = add(gi[2 * y], mul(r, sub(gi[2 * y + 1], gi[2 * y])));
            }
        }
        if (si + 1 == dev.stages().size())
            for (int i = 0; i < M; i++) {   // nothing is left to sum over: the folded sums are the reveals f_i(R)
                h_f_evals[2 * i] = g[(size_t)i * size].c0;
                h_f_evals[2 * i + 1] = g[(size_t)i * size].c1;
            }
    }
    Dot fin;
    for (int i = 0; i < M; i++) {
        t.append_ext2(SP_LABEL(L_FEVAL), h_f_evals[2 * i], h_f_evals[2 * i + 1]);
        fin.mac(scale[i], E2{h_f_evals[2 * i], h_f_evals[2 * i + 1]});   // scale_i = alpha^i eq(r_i, R)
    }
    const E2 v = fin.value();
    h_final_eval[0] = v.c0;
    h_final_eval[1] = v.c1;
    return MB_OK;
}

// The rounds on the values of their polynomial over all leaves.
int rounds_by_share(SamePointDevice& dev, int M, int arity, E2 alpha, AglTranscript& t, uint64_t* h_round_msgs, uint64_t* h_challenges,
                    uint64_t* h_f_evals, uint64_t* h_final_eval) {
    std::vector<E2> R(arity), u(sp::SHARE);
    for (size_t si = 0; si < dev.stages().size(); si++) {
        const Stage st = dev.stages()[si];
        int rc;
        if (si > 0) {
            // the challenges that the pass consumes: all of a word's for the first extension table
            const int from = st.source == FROM_WORDS ? 0 : dev.stages()[si - 1].first;
            rc = dev.fold(si, R.data() + from, st.first - from);
        } else {
            rc = dev.first_share(alpha);
        }
        if (rc != MB_OK) return rc;
        t.begin_append(SP_LABEL(L_MSG));   // while the pass runs
        rc = dev.wait();
        if (rc != MB_OK) return rc;
        int size = 1;
        for (int j = 0; j < st.rounds; j++) size *= 3;
        for (int x = 0; x < size; x++) u[x] = E2{dev.values()[2 * x], dev.values()[2 * x + 1]};
        for (int j = 0; j < st.rounds; j++) {
            // q0 (1 - c) + q1 c + q2 (c^2 - c): the sums over the later variables at 0 and 1
            const int round = st.first + j, rest = size / 3, later = st.rounds - j - 1;
            E2 q[3] = {E2{0, 0}, E2{0, 0}, E2{0, 0}};
            for (int m = 0; m < (1 << later); m++) {
                int at = 0, digit = 1;
                for (int b = 0; b < later; b++, digit *= 3) at += ((m >> b) & 1) * digit;
                for (int p = 0; p < 3; p++) q[p] = add(q[p], u[3 * at + p]);
            }
            const E2 q12 = add(q[1], q[2]), msg[3] = {q[0], q[1], sub(add(q12, q12), q[0])};
            for (int c = 0; c < 3; c++) {
                if (c > 0 || j > 0) t.begin_append(SP_LABEL(L_MSG));
                t.finish_append_ext2(msg[c].c0, msg[c].c1);
                h_round_msgs[((size_t)round * 3 + c) * 2] = msg[c].c0;
                h_round_msgs[((size_t)round * 3 + c) * 2 + 1] = msg[c].c1;
            }
            const E2 r = challenge(t, SP_LABEL(L_CH));
            R[round] = r;
            if (h_challenges) { h_challenges[2 * round] = r.c0; h_challenges[2 * round + 1] = r.c1; }
            const E2 rr = sub(mul(r, r), r);
            for (int y = 0; y < rest; y++)
                u[y] = add(add(u[3 * y], mul(r, sub(u[3 * y + 1], u[3 * y]))), mul(rr, u[3 * y + 2]));
            size = rest;
        }
    }
    // nothing is left to sum over: the last stage's sums, folded, are the reveals f_i(R), and what is left of the polynomial is
    // sum_i alpha^i eq(r_i, R) f_i(R)
    const Stage end = dev.stages().back();
    for (int i = 0; i < M; i++) {
        E2 g[1 << sp::MAX_B];
        for (int m = 0; m < (1 << end.rounds); m++) g[m] = ld(dev.sums() + 2 * (((size_t)i << end.rounds) + m));
        for (int j = 0; j < end.rounds; j++)
            for (int m = 0; m < (1 << (end.rounds - j - 1)); m++)
                g[m] = add(g[2 * m], mul(R[end.first + j], sub(g[2 * m + 1], g[2 * m])));
        h_f_evals[2 * i] = g[0].c0;
        h_f_evals[2 * i + 1] = g[0].c1;
        t.append_ext2(SP_LABEL(L_FEVAL), g[0].c0, g[0].c1);
    }
    h_final_eval[0] = u[0].c0;
    h_final_eval[1] = u[0].c1;
    return MB_OK;
}

}  // namespace

// kind 0: d_w0 = packed bits [M][words]; 1: d_w0 / d_w1 = +1 / -1 masks [M][words]; 2: d_w0 = extension tables
// [M][2^arity][2]. words = max(1, 2^(arity - 6)).
int same_point_prove(int M, int arity, const uint64_t* h_pts, const uint64_t* h_vals, int kind, const uint64_t* d_w0,
                     const uint64_t* d_w1, AglTranscript& t, uint64_t* h_round_msgs, uint64_t* h_challenges, uint64_t* h_f_evals,
                     uint64_t* h_final_eval) {
    if (M < 1 || M > 4096 || arity < 1 || arity > 32 || !h_pts || !h_vals || !d_w0 || kind < 0 || kind > 2 || (kind == 1 && !d_w1) ||
        !h_round_msgs || !h_f_evals || !h_final_eval)
        return MB_ERR_ARG;
    // the first pass does not depend on alpha: it is queued first, and the header of the transcript (every claim
    // point, label by label) is absorbed while the device works
    const bool share = M * arity >= SHARE_FROM;
    SamePointDevice dev;
    int rc = dev.init(M, arity, h_pts, kind, d_w0, d_w1, false, share);
    if (rc != MB_OK) return rc;
    header(t, M, arity, h_pts, h_vals);
    const E2 alpha = challenge(t, SP_LABEL(L_ALPHA));
    return !share ? rounds_by_leaf(dev, M, arity, h_pts, alpha, t, h_round_msgs, h_challenges, h_f_evals, h_final_eval)
                          : rounds_by_share(dev, M, arity, alpha, t, h_round_msgs, h_challenges, h_f_evals, h_final_eval);
}

// verify_same_point for instances of any arity <= num_vars: pts are concatenated (arity[i] pairs each).
int same_point_verify(int M, int N, const int* arity, const uint64_t* h_pts, const uint64_t* h_vals, const uint64_t* round_msgs,
                      const uint64_t* f_evals, const uint64_t* final_eval, AglTranscript& t, uint64_t* challenges, int* ok) {
    *ok = 0;
    if (M < 1 || N < 1 || N > 62) return MB_ERR_ARG;
    t.append_u64(SP_LABEL(L_NUM_VAR), (uint64_t)N);
    t.append_u64(SP_LABEL(L_NUM_INST), (uint64_t)M);
    std::vector<size_t> off(M);
    size_t o = 0;
    for (int i = 0; i < M; i++) {
        if (arity[i] < 0 || arity[i] > N) return MB_ERR_ARG;
        off[i] = o;
        t.append_u64(SP_LABEL(L_ARITY), (uint64_t)arity[i]);
        for (int k = 0; k < arity[i]; k++) t.append_ext2(SP_LABEL(L_R), h_pts[o + 2 * k], h_pts[o + 2 * k + 1]);
        t.append_ext2(SP_LABEL(L_Y), h_vals[2 * i], h_vals[2 * i + 1]);
        o += 2 * (size_t)arity[i];
    }
    const E2 alpha = challenge(t, SP_LABEL(L_ALPHA));
    std::vector<E2> alphas(M), R(N);
    E2 pw{1, 0}, current{0, 0};
    for (int i = 0; i < M; i++) {
        alphas[i] = pw;
        pw = e2c(agl::e2_mul(pw, alpha));
        const E2 weight{(uint64_t)1 << (N - arity[i]), 0};
        current = agl::e2_add(current, agl::e2_mul(alphas[i], e2c(agl::e2_mul(ld(h_vals + 2 * i), weight))));
    }
    current = e2c(current);
    const E2 inv2 = e2c(agl::e2_inv(E2{2, 0})), one{1, 0}, two{2, 0};
    for (int round = 0; round < N; round++) {
        E2 m[3];
        for (int c = 0; c < 3; c++) m[c] = ld(round_msgs + ((size_t)round * 3 + c) * 2);
        const E2 sum = e2c(agl::e2_add(m[0], m[1]));
        if (sum.c0 != current.c0 || sum.c1 != current.c1) return MB_OK;
        for (int c = 0; c < 3; c++) t.append_ext2(SP_LABEL(L_MSG), m[c].c0, m[c].c1);
        const E2 r = challenge(t, SP_LABEL(L_CH));
        R[round] = r;
        if (challenges) { challenges[2 * round] = r.c0; challenges[2 * round + 1] = r.c1; }
        // Lagrange through 0, 1, 2 (same_point_sumcheck.rs:886-904)
        const E2 xm1 = agl::e2_sub(r, one), xm2 = agl::e2_sub(r, two);
        const E2 l0 = agl::e2_mul(e2c(agl::e2_mul(xm1, xm2)), inv2);
        const E2 l1 = agl::e2_sub(E2{0, 0}, agl::e2_mul(r, xm2));
        const E2 l2 = agl::e2_mul(e2c(agl::e2_mul(r, xm1)), inv2);
        current = e2c(agl::e2_add(agl::e2_add(agl::e2_mul(e2c(l0), m[0]), agl::e2_mul(e2c(l1), m[1])), agl::e2_mul(e2c(l2), m[2])));
    }
    E2 expected{0, 0};
    for (int i = 0; i < M; i++) t.append_ext2(SP_LABEL(L_FEVAL), f_evals[2 * i], f_evals[2 * i + 1]);
    for (int i = 0; i < M; i++) {
        const E2 eq_i = eq_eval(h_pts + off[i], R.data(), arity[i]);
        expected = agl::e2_add(expected, agl::e2_mul(alphas[i], e2c(agl::e2_mul(eq_i, ld(f_evals + 2 * i)))));
    }
    expected = e2c(expected);
    const E2 fin = ld(final_eval);
    *ok = current.c0 == expected.c0 && current.c1 == expected.c1 && fin.c0 == expected.c0 && fin.c1 == expected.c1;
    return MB_OK;
}

}  // namespace mbhost

extern "C" {

// The whole same-point sumcheck for num_leaves instances of one arity (the reference's device path,
// same_point_sumcheck.rs:1334-1553). h_claim_pts[num_leaves][arity][2], h_claim_vals[num_leaves][2]; witness on the
// device: kind 0 binary packed (d_w0[num_leaves][words], words = max(1, 2^(arity - 6))), 1 ternary single chunk
// (d_w0 = +1 masks, d_w1 = -1 masks), 2 extension tables (d_w0[num_leaves][2^arity][2]). `transcript`: a handle
// from agl_transcript_create, advanced by the proof. Host outputs: round_msgs[arity][3][2], challenges[arity][2]
// (may be null), f_evals[num_leaves][2], final_eval[2]. Device memory beyond the caller's: about
// num_leaves x 2^(arity - 6) x 17 bytes for packed witnesses, num_leaves x 2^(arity - 4) x 17 for extension tables.
int agl_same_point_prove_device_ffi(int num_leaves, int arity, const uint64_t* h_claim_pts, const uint64_t* h_claim_vals, int kind,
                                    const uint64_t* d_w0, const uint64_t* d_w1, void* transcript, uint64_t* h_round_msgs,
                                    uint64_t* h_challenges, uint64_t* h_f_evals, uint64_t* h_final_eval) {
    if (!transcript) return MB_ERR_ARG;
    return mbhost::same_point_prove(num_leaves, arity, h_claim_pts, h_claim_vals, kind, d_w0, d_w1,
                                    *static_cast<mbhost::AglTranscript*>(transcript), h_round_msgs, h_challenges, h_f_evals,
                                    h_final_eval);
}

// The claims y_i = f_i(r_i) of the leaves (the witness' multilinear extension at its claim point), computed on the
// device with the kernels of the proof: h_claim_vals[num_leaves][2]. Arguments as agl_same_point_prove_device_ffi.
int agl_same_point_claims_device_ffi(int num_leaves, int arity, const uint64_t* h_claim_pts, int kind, const uint64_t* d_w0,
                                     const uint64_t* d_w1, uint64_t* h_claim_vals) {
    return mbhost::same_point_claims(num_leaves, arity, h_claim_pts, kind, d_w0, d_w1, h_claim_vals);
}

// verify_same_point on the host (same_point_sumcheck.rs:161-219); instances may have different arities
// (h_claim_pts holds arity[i] pairs per instance, back to back). *ok = 1 when the proof is accepted; the
// challenges (num_vars pairs) are written when `challenges` is not null.
int agl_same_point_verify_ffi(int num_instances, int num_vars, const int* arity, const uint64_t* h_claim_pts,
                              const uint64_t* h_claim_vals, const uint64_t* round_msgs, const uint64_t* f_evals,
                              const uint64_t* final_eval, void* transcript, uint64_t* challenges, int* ok) {
    if (!transcript || !ok || !arity || !h_claim_pts || !h_claim_vals || !round_msgs || !f_evals || !final_eval) return MB_ERR_ARG;
    return mbhost::same_point_verify(num_instances, num_vars, arity, h_claim_pts, h_claim_vals, round_msgs, f_evals, final_eval,
                                     *static_cast<mbhost::AglTranscript*>(transcript), challenges, ok);
}

}  // extern "C"
