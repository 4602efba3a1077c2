// Host layer for the batched degree-3 sumcheck (shared eq table, K instances
// combined with powers of alpha) over Goldilocks, one shard of the hypercube.
//
// A shard holds the slice of every table whose top index bits equal the shard
// number: a_k, b_k slices of 2^n_loc base-field elements, and the eq slice
// eq(t_low, x_low) * eq(t_top, shard) (the scalar is passed in). The per-round
// API mirrors the reference's state objects (compute message, then fold on the
// challenge; almost-goldilocks-cuda-rs/src/sumcheck_prover.rs:127-436): the
// caller adds the shards' messages, runs the transcript and broadcasts the
// challenge. With one shard it is the whole prover. The C-ABI below also exposes
// the host transcript (zk-torch-3/src/transcript.rs:174-350) so that callers in
// any language run the same Fiat-Shamir.
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "exchange.hpp"
#include "gl_transcript.hpp"
#include "../gl_sumcheck_launch.cuh"
#include "pair_sumcheck.cuh"

using namespace mb;
using namespace mb::sc;

namespace mbhost {

constexpr int BATCHED_MAX_K = 64;

// The round polynomials of sum_x eq(t, x) sum_k alpha^k a_k(x) b_k(x) factor: m(c) = lambda(c) T(c) with
// lambda(c) = (1 - t_i) + c (2 t_i - 1) times the eq value of the variables bound before, and T quadratic. T comes from
// the several-rounds-per-pass engine (pair_sumcheck.cuh): the first pass is independent of alpha and gives every
// instance its own matrix, from which the claims are read and, once alpha is known, the first rounds run; the eq table
// (as large as an instance) is never formed.
class BatchedEqAbState {
public:
    using Pair = PairSumcheck<pr::GlF, PairGl>;
    using H = PairHost<pr::GlF, PairGl>;
    using E2 = gl::E2;

    // threads: the handle may be used from other host threads than this one, so every call ends with the work it
    // queued (another thread's stream knows nothing of this one's)
    int init(const uint64_t* d_a, const uint64_t* d_b, const uint64_t* h_point_low, const uint64_t* h_eq_scale, int K,
             int n_loc, bool threads) {
        if (!d_a || !d_b || !h_eq_scale || K < 1 || K > BATCHED_MAX_K || n_loc < 1 || n_loc > 34) return MB_ERR_ARG;
        if (!h_point_low || !aligned16(d_a) || !aligned16(d_b)) return MB_ERR_ARG;
        K_ = K; n_loc_ = n_loc; threads_ = threads;
        shard_ = H::canon(E2{h_eq_scale[0], h_eq_scale[1]});
        // the caller's base-field tables are read in place until the first fold and never written
        int rc = pair_.init(d_a, d_b, (size_t)1 << n_loc, K, n_loc, true, h_point_low, n_loc);
        return rc == MB_OK ? finish_call() : rc;
    }
    // Local share of the per-instance claims sum_x eq a_k b_k (K extension elements), whatever round the state is in: they
    // are read off the first pass, which the folds overwrite, so the first fold keeps them.
    int claims(uint64_t* h_out) {
        int rc = keep_claims();
        if (rc != MB_OK) return rc;
        for (int k = 0; k < K_; k++) {
            h_out[2 * k] = claims_[k].c0;
            h_out[2 * k + 1] = claims_[k].c1;
        }
        return MB_OK;
    }
    // Counts until the first fold, which combines the instances; later calls change nothing.
    int set_alpha(Ext2 alpha) {
        if (round_ > 0) return MB_OK;
        alphas_.resize(K_);
        E2 p{1, 0};
        const E2 a = H::canon(E2{alpha.c0, alpha.c1});
        for (int k = 0; k < K_; k++) {
            alphas_[k] = p;
            p = H::mul(p, a);
        }
        return pair_.set_scale(alphas_.data());
    }
    // Local share of m(0..3) for the current round: T(2) = 2 T(1) + 2 T2 - T(0), T(3) = 3 T(1) + 6 T2 - 2 T(0).
    int round_message(uint64_t* h_msg) {
        if (alphas_.empty() || round_ >= n_loc_) return MB_ERR_ARG;
        E2 t0, t1, t2;
        int rc = pair_.sums(t0, t1, t2);
        if (rc != MB_OK) return rc;
        const E2 s12 = H::add(t1, t2), d = H::sub(H::add(s12, s12), t0);      // T(2)
        const E2 t22 = H::add(t2, t2), s = H::add(H::sub(H::add(d, t1), t0), H::add(t22, t22));   // T(3)
        const E2 T[4] = {t0, t1, d, s};
        const E2 t = pair_.eq_coord(round_), one{1, 0}, w = H::mul(shard_, pair_.eq_scale());
        E2 lam = H::mul(w, H::sub(one, t));
        const E2 step = H::mul(w, H::sub(H::add(t, t), one));
        for (int c = 0; c < 4; c++) {
            const E2 m = H::mul(lam, T[c]);
            h_msg[2 * c] = m.c0;
            h_msg[2 * c + 1] = m.c1;
            lam = H::add(lam, step);
        }
        return MB_OK;
    }
    int fold(Ext2 ch) {
        if (alphas_.empty() || round_ >= n_loc_) return MB_ERR_ARG;
        int rc = round_ == 0 ? keep_claims() : MB_OK;
        if (rc != MB_OK) return rc;
        round_++;
        rc = pair_.fold(H::canon(E2{ch.c0, ch.c1}));
        return rc == MB_OK ? finish_call() : rc;
    }
    // After n_loc folds: eq (with the shard's factor), a_k, b_k: (2K + 1) extension elements; scaled: alpha^k a_k.
    int finals(uint64_t* h_out, bool scaled) {
        if (round_ != n_loc_) return MB_ERR_ARG;
        std::vector<E2> v(2 * (size_t)K_ + 1);
        v[0] = H::mul(shard_, pair_.eq_scale());
        int rc = pair_.finals(v.data() + 1, v.data() + 1 + K_);
        if (rc != MB_OK) return rc;
        for (int k = 0; k < K_ && scaled; k++) v[1 + k] = H::mul(alphas_[k], v[1 + k]);
        for (size_t i = 0; i < v.size(); i++) {
            h_out[2 * i] = v[i].c0;
            h_out[2 * i + 1] = v[i].c1;
        }
        return MB_OK;
    }

private:
    int keep_claims() {
        if (!claims_.empty()) return MB_OK;
        std::vector<E2> c(K_);
        int rc = pair_.claims(c.data());
        if (rc != MB_OK) return rc;
        for (E2& v : c) v = H::mul(v, shard_);
        claims_.swap(c);
        return MB_OK;
    }
    int finish_call() {
        if (threads_) MB_CUDA(cudaStreamSynchronize(MB_STREAM));
        return MB_OK;
    }
    int K_ = 0, n_loc_ = 0, round_ = 0;
    bool threads_ = false;
    E2 shard_{1, 0};
    std::vector<E2> alphas_, claims_;
    Pair pair_;
};

}  // namespace mbhost


// ---- one proof over `world` shards: round loop, recombination, transcript and the last log2(world) rounds ----
namespace {

using gl::E2;
inline E2 e2c(E2 a) { return gl::e2_canon(a); }
inline E2 e2_load(const uint64_t* w) { return E2{gl::canon(w[0]), gl::canon(w[1])}; }

// Sum over the ranks of `width` extension elements each (rank-major words).
void sum_shares(const uint64_t* all, int world, int width, E2* out) {
    for (int i = 0; i < width; i++) {
        E2 t{0, 0};
        for (int g = 0; g < world; g++) t = gl::e2_add(t, e2_load(all + ((size_t)g * width + i) * 2));
        out[i] = e2c(t);
    }
}

struct RoundClock {
    bool on = std::getenv("MB_SHARD_TIMING") != nullptr;
    std::chrono::steady_clock::time_point t0;
    double kernel = 0, gather = 0, host = 0;
    void start() { if (on) t0 = std::chrono::steady_clock::now(); }
    void stop(double& acc) {
        if (!on) return;
        auto t1 = std::chrono::steady_clock::now();
        acc += std::chrono::duration<double, std::micro>(t1 - t0).count();
        t0 = t1;
    }
};

}  // namespace

namespace mbhost {

// Every rank passes its slices; all outputs are identical on every rank.
int batched_prove_sharded(const mb_exchange* ex, const uint64_t* d_a, const uint64_t* d_b, int K, int num_vars,
                          const uint64_t* h_point, const uint8_t* label, size_t label_len, uint64_t* h_claims,
                          uint64_t* h_alpha, uint64_t* h_round_msgs, uint64_t* h_challenges, uint64_t* h_finals,
                          uint64_t* h_final_eval, uint64_t* h_transcript_state, double* h_round_us) {
    if (!ex || !d_a || !d_b || !h_point || (!label && label_len) || K < 1 || K > BATCHED_MAX_K) return MB_ERR_ARG;
    const int world = ex->world, rank = ex->rank;
    int g_bits = 0;
    while ((1 << g_bits) < world) g_bits++;
    if (world < 1 || (1 << g_bits) != world || rank < 0 || rank >= world) return MB_ERR_ARG;
    const int n_loc = num_vars - g_bits;
    if (n_loc < 1 || n_loc > 34) return MB_ERR_UNSUPPORTED;

    // eq(t_top, rank): bit i of the rank pairs with coordinate n_loc + i
    E2 scale{1, 0};
    for (int i = 0; i < g_bits; i++) {
        const E2 t = e2_load(h_point + 2 * (size_t)(n_loc + i));
        scale = e2c(gl::e2_mul(scale, (rank >> i) & 1 ? t : gl::e2_sub(E2{1, 0}, t)));
    }
    const uint64_t scale_w[2] = {scale.c0, scale.c1};

    BatchedEqAbState st;
    int rc = st.init(d_a, d_b, h_point, scale_w, K, n_loc, false);
    if (rc != MB_OK) return rc;

    using H = BatchedEqAbState::H;
    const int T = 2 * K + 1;
    std::vector<uint64_t> mine((size_t)2 * (T > 4 ? T : 4)), all((size_t)world * mine.size());
    std::vector<E2> claims(K);
    Transcript tr(label, label_len);
    tr.append_u64("sp_num_var", (uint64_t)num_vars);
    tr.append_u64("sp_num_inst", (uint64_t)K);
    rc = st.claims(mine.data());
    if (rc != MB_OK) return rc;
    rc = ex->all_gather_host(ex->ctx, mine.data(), 2 * (size_t)K, all.data());
    if (rc != MB_OK) return rc;
    sum_shares(all.data(), world, K, claims.data());
    for (int k = 0; k < K; k++) {
        tr.append_ext2("sp_y_i", Ext2{claims[k].c0, claims[k].c1});
        if (h_claims) { h_claims[2 * k] = claims[k].c0; h_claims[2 * k + 1] = claims[k].c1; }
    }
    const Ext2 alpha = tr.challenge_ext2("sp_alpha");
    if (h_alpha) { h_alpha[0] = alpha.c0; h_alpha[1] = alpha.c1; }
    rc = st.set_alpha(alpha);
    if (rc != MB_OK) return rc;

    RoundClock clock;
    int round = 0;
    bool label_absorbed = false;   // the first label of a round goes in while the round's kernel runs
    auto publish = [&](const E2* msg) {
        for (int c = 0; c < 4; c++) {
            if (c > 0 || !label_absorbed) tr.begin_append("sp_round_msg");
            tr.finish_append_ext2(Ext2{msg[c].c0, msg[c].c1});
            if (h_round_msgs) {
                h_round_msgs[(size_t)round * 8 + 2 * c] = msg[c].c0;
                h_round_msgs[(size_t)round * 8 + 2 * c + 1] = msg[c].c1;
            }
        }
        const Ext2 r = tr.challenge_ext2("sp_round_challenge");
        if (h_challenges) { h_challenges[2 * (size_t)round] = r.c0; h_challenges[2 * (size_t)round + 1] = r.c1; }
        round++;
        label_absorbed = false;
        return r;
    };
    for (int i = 0; i < n_loc; i++) {
        clock.start();
        rc = st.round_message(mine.data());
        if (rc != MB_OK) return rc;
        clock.stop(clock.kernel);
        E2 msg[4];
        if (world > 1) {
            rc = ex->all_gather_host(ex->ctx, mine.data(), 8, all.data());
            if (rc != MB_OK) return rc;
            clock.stop(clock.gather);
            sum_shares(all.data(), world, 4, msg);
        } else {
            for (int c = 0; c < 4; c++) msg[c] = e2_load(mine.data() + 2 * c);
        }
        const Ext2 r = publish(msg);
        clock.stop(clock.host);
        rc = st.fold(r);
        if (rc != MB_OK) return rc;
        if (round < num_vars) {
            tr.begin_append("sp_round_msg");
            label_absorbed = true;
        }
    }
    // one value per table and rank: eq, a_k, b_k; the top variables are finished on the host
    clock.start();
    rc = st.finals(mine.data(), false);
    if (rc != MB_OK) return rc;
    clock.stop(clock.kernel);
    rc = ex->all_gather_host(ex->ctx, mine.data(), 2 * (size_t)T, all.data());
    if (rc != MB_OK) return rc;
    clock.stop(clock.gather);
    std::vector<std::vector<E2>> tab(T, std::vector<E2>(world));
    for (int g = 0; g < world; g++)
        for (int i = 0; i < T; i++) tab[i][g] = e2_load(all.data() + ((size_t)g * T + i) * 2);
    std::vector<E2> alphas(K);
    {
        E2 pw{1, 0};
        for (int k = 0; k < K; k++) {
            alphas[k] = pw;
            pw = H::mul(pw, E2{alpha.c0, alpha.c1});
        }
    }
    for (int size = world; size > 1; size /= 2) {
        const int half = size / 2;
        E2 msg[4];
        for (int c = 0; c < 4; c++) {
            const E2 cc{(uint64_t)c, 0};
            E2 tot{0, 0};
            for (int y = 0; y < half; y++) {
                auto at = [&](const std::vector<E2>& t) {
                    return e2c(gl::e2_add(t[2 * y], gl::e2_mul(cc, gl::e2_sub(t[2 * y + 1], t[2 * y]))));
                };
                E2 inner{0, 0};
                for (int k = 0; k < K; k++)
                    inner = gl::e2_add(inner, gl::e2_mul(alphas[k], e2c(gl::e2_mul(at(tab[1 + k]), at(tab[1 + K + k])))));
                tot = gl::e2_add(tot, gl::e2_mul(at(tab[0]), e2c(inner)));
            }
            msg[c] = e2c(tot);
        }
        const Ext2 rr = publish(msg);
        const E2 r{rr.c0, rr.c1};
        for (auto& t : tab)
            for (int y = 0; y < half; y++) t[y] = e2c(gl::e2_add(t[2 * y], gl::e2_mul(r, gl::e2_sub(t[2 * y + 1], t[2 * y]))));
    }
    std::vector<E2> fin(T);
    E2 acc{0, 0};
    for (int i = 0; i < T; i++) fin[i] = tab[i][0];
    for (int k = 0; k < K; k++) acc = H::add(acc, H::mul(alphas[k], H::mul(fin[1 + k], fin[1 + K + k])));
    for (int i = 0; i < T; i++) {
        tr.append_ext2("sp_f_eval", Ext2{fin[i].c0, fin[i].c1});
        if (h_finals) { h_finals[2 * i] = fin[i].c0; h_finals[2 * i + 1] = fin[i].c1; }
    }
    const E2 fe = H::mul(fin[0], acc);
    if (h_final_eval) { h_final_eval[0] = fe.c0; h_final_eval[1] = fe.c1; }
    if (h_transcript_state) std::memcpy(h_transcript_state, tr.state(), 64);
    clock.stop(clock.host);
    if (h_round_us) {
        // what the local rounds cost besides their kernels, per round: exchange, recombination and transcript
        h_round_us[0] = clock.on ? clock.kernel / (n_loc + 1) : -1.0;
        h_round_us[1] = clock.on ? clock.gather / (n_loc + 1) : -1.0;
        h_round_us[2] = clock.on ? clock.host / (n_loc + 1) : -1.0;
    }
    return MB_OK;
}

}  // namespace mbhost

using mbhost::BatchedEqAbState;
using mbhost::Ext2;
using mbhost::Transcript;

extern "C" {

// ---- one shard of the batched eq * a_k * b_k sumcheck ----
// d_a, d_b: [K][2^n_loc] base-field slices (read in place until the first fold, never written); h_point_low: n_loc (c0, c1) pairs (the
// shard-local coordinates of the eq point); h_eq_scale: eq of the top coordinates
// at this shard's index ((1, 0) for a single shard).
int gl_batched_state_create(const uint64_t* d_a, const uint64_t* d_b, const uint64_t* h_point_low,
                            const uint64_t* h_eq_scale, int K, int n_loc, void** state) {
    if (!state) return MB_ERR_ARG;
    auto* s = new BatchedEqAbState;
    int rc = s->init(d_a, d_b, h_point_low, h_eq_scale, K, n_loc, true);
    if (rc != MB_OK) { delete s; return rc; }
    *state = s;
    return MB_OK;
}
int gl_batched_state_destroy(void* state) { delete static_cast<BatchedEqAbState*>(state); return MB_OK; }
int gl_batched_state_claims(void* state, uint64_t* h_claims) { return static_cast<BatchedEqAbState*>(state)->claims(h_claims); }
int gl_batched_state_set_alpha(void* state, uint64_t c0, uint64_t c1) { return static_cast<BatchedEqAbState*>(state)->set_alpha(Ext2{c0, c1}); }
int gl_batched_state_round_message(void* state, uint64_t* h_msg) { return static_cast<BatchedEqAbState*>(state)->round_message(h_msg); }
int gl_batched_state_fold(void* state, uint64_t c0, uint64_t c1) { return static_cast<BatchedEqAbState*>(state)->fold(Ext2{c0, c1}); }
int gl_batched_state_finals(void* state, uint64_t* h_out) { return static_cast<BatchedEqAbState*>(state)->finals(h_out, true); }

// ---- the whole proof over the shards of an exchange (world = 1: an mb_exchange_local_create(1) object) ----
// d_a, d_b: this rank's slices [K][2^(num_vars - log2 world)]; h_point: num_vars (c0, c1) pairs, the same on every
// rank. Outputs (each may be null), identical on every rank: claims [K][2], alpha [2], round messages
// [num_vars][4][2], challenges [num_vars][2], finals [2K + 1][2] (eq, a_k, b_k at the challenge point), final
// evaluation [2], transcript state [8]; h_round_us [3]: with MB_SHARD_TIMING set, microseconds per local round spent
// waiting for the kernel, in the exchange, and on the host (recombination and transcript); -1 otherwise.
int gl_batched_prove_sharded(const mb_exchange* ex, const uint64_t* d_a, const uint64_t* d_b, int K, int num_vars,
                             const uint64_t* h_point, const uint8_t* label, size_t label_len, uint64_t* h_claims,
                             uint64_t* h_alpha, uint64_t* h_round_msgs, uint64_t* h_challenges, uint64_t* h_finals,
                             uint64_t* h_final_eval, uint64_t* h_transcript_state, double* h_round_us) {
    return mbhost::batched_prove_sharded(ex, d_a, d_b, K, num_vars, h_point, label, label_len, h_claims, h_alpha, h_round_msgs,
                                         h_challenges, h_finals, h_final_eval, h_transcript_state, h_round_us);
}

// ---- host transcript ----
int gl_transcript_create(const uint8_t* label, size_t label_len, void** transcript) {
    if (!transcript) return MB_ERR_ARG;
    *transcript = new Transcript(label, label_len);
    return MB_OK;
}
int gl_transcript_destroy(void* t) { delete static_cast<Transcript*>(t); return MB_OK; }
int gl_transcript_append_u64(void* t, const char* label, uint64_t v) { static_cast<Transcript*>(t)->append_u64(label, v); return MB_OK; }
int gl_transcript_append_ext2(void* t, const char* label, uint64_t c0, uint64_t c1) {
    static_cast<Transcript*>(t)->append_ext2(label, Ext2{c0, c1});
    return MB_OK;
}
int gl_transcript_challenge_ext2(void* t, const char* label, uint64_t* out2) {
    Ext2 r = static_cast<Transcript*>(t)->challenge_ext2(label);
    out2[0] = r.c0;
    out2[1] = r.c1;
    return MB_OK;
}
int gl_transcript_state(const void* t, uint64_t* out8) { std::memcpy(out8, static_cast<const Transcript*>(t)->state(), 64); return MB_OK; }

// Verifier of the batched eq * a * b proof on the host (no device call): replays the transcript of
// gl_batched_prove_sharded, checks P(0) + P(1) against the running claim in every round (the first claim is
// sum_k alpha^k y_k), takes P(r) by interpolation on 0..3 as the next claim, and at the end checks that the last
// claim equals eq(R) sum_k alpha^k a_k(R) b_k(R) and that the revealed eq(R) is the eq polynomial of h_point at the
// challenges (round i binds variable i). The revealed a_k(R), b_k(R) are the openings the caller checks against its
// commitments. h_claims [K][2], h_round_msgs [num_vars][4][2], h_finals [2K + 1][2]; h_challenges [num_vars][2]
// (may be null) receives the challenges. *ok = 1 when accepted.
int gl_batched_verify_host(int K, int num_vars, const uint64_t* h_point, const uint8_t* label, size_t label_len,
                           const uint64_t* h_claims, const uint64_t* h_round_msgs, const uint64_t* h_finals,
                           uint64_t* h_challenges, int* ok) {
    using namespace mbhost;
    if (K < 1 || num_vars < 1 || num_vars > 40 || !h_point || !h_claims || !h_round_msgs || !h_finals || !ok || (!label && label_len))
        return MB_ERR_ARG;
    *ok = 0;
    Transcript tr(label, label_len);
    tr.append_u64("sp_num_var", (uint64_t)num_vars);
    tr.append_u64("sp_num_inst", (uint64_t)K);
    for (int k = 0; k < K; k++) tr.append_ext2("sp_y_i", Ext2{gl::canon(h_claims[2 * k]), gl::canon(h_claims[2 * k + 1])});
    const Ext2 a = tr.challenge_ext2("sp_alpha");
    const E2 alpha{a.c0, a.c1};
    E2 claim{0, 0}, pw{1, 0};
    for (int k = 0; k < K; k++) {
        claim = e2c(gl::e2_add(claim, gl::e2_mul(pw, e2_load(h_claims + 2 * k))));
        pw = e2c(gl::e2_mul(pw, alpha));
    }
    // 1 / ((c - 0)(c - 1)...(c - 3)) without the factor c - c, for c = 0..3: -1/6, 1/2, -1/2, 1/6
    const uint64_t inv2 = gl::canon(gl::inv(2)), inv6 = gl::canon(gl::inv(6));
    const uint64_t wgt[4] = {gl::canon(gl::sub(0, inv6)), inv2, gl::canon(gl::sub(0, inv2)), inv6};
    E2 eq_at_r{1, 0};
    for (int round = 0; round < num_vars; round++) {
        E2 msg[4];
        for (int c = 0; c < 4; c++) msg[c] = e2_load(h_round_msgs + (size_t)round * 8 + 2 * c);
        const E2 sum = e2c(gl::e2_add(msg[0], msg[1]));
        if (sum.c0 != claim.c0 || sum.c1 != claim.c1) return MB_OK;
        for (int c = 0; c < 4; c++) tr.append_ext2("sp_round_msg", Ext2{msg[c].c0, msg[c].c1});
        const Ext2 rr = tr.challenge_ext2("sp_round_challenge");
        const E2 r{rr.c0, rr.c1};
        if (h_challenges) { h_challenges[2 * round] = r.c0; h_challenges[2 * round + 1] = r.c1; }
        // P(r) = sum_c P(c) w_c prod_{k != c} (r - k)
        E2 next{0, 0};
        for (int c = 0; c < 4; c++) {
            E2 num{wgt[c], 0};
            for (int k = 0; k < 4; k++)
                if (k != c) num = e2c(gl::e2_mul(num, gl::e2_sub(r, E2{(uint64_t)k, 0})));
            next = gl::e2_add(next, gl::e2_mul(msg[c], num));
        }
        claim = e2c(next);
        // eq factor of variable `round`: p r + (1 - p)(1 - r)
        const E2 p = e2_load(h_point + 2 * round), one{1, 0};
        const E2 f = gl::e2_add(gl::e2_mul(p, r), gl::e2_mul(gl::e2_sub(one, p), gl::e2_sub(one, r)));
        eq_at_r = e2c(gl::e2_mul(eq_at_r, e2c(f)));
    }
    const int T = 2 * K + 1;
    for (int i = 0; i < T; i++) tr.append_ext2("sp_f_eval", Ext2{gl::canon(h_finals[2 * i]), gl::canon(h_finals[2 * i + 1])});
    const E2 eq_rev = e2_load(h_finals);
    if (eq_rev.c0 != eq_at_r.c0 || eq_rev.c1 != eq_at_r.c1) return MB_OK;
    E2 acc{0, 0};
    pw = E2{1, 0};
    for (int k = 0; k < K; k++) {
        acc = e2c(gl::e2_add(acc, gl::e2_mul(pw, e2c(gl::e2_mul(e2_load(h_finals + 2 * (1 + k)), e2_load(h_finals + 2 * (1 + K + k)))))));
        pw = e2c(gl::e2_mul(pw, alpha));
    }
    const E2 last = e2c(gl::e2_mul(eq_rev, acc));
    *ok = last.c0 == claim.c0 && last.c1 == claim.c1;
    return MB_OK;
}


}  // extern "C"
