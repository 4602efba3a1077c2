// Host layer above the C-ABI for the almost-Goldilocks sumcheck: the prover loop
// and the verifier the reference keeps in Rust (zk-torch-4), written in C++
// because no Rust toolchain exists on the build machine.
//
//   GpuLinearSumcheckProver::new / prove / prove_ext2 / prove_gpu_resident
//                                     zk-torch-4/src/sumcheck/gpu_prover.rs:26-112
//   CpuLinearSumcheckProverExt2       zk-torch-4/src/sumcheck/cpu_ext2_prover.rs:21-100
//                                     (same transcript labels, interoperable proofs)
//   SumcheckVerifier::verify          zk-torch-4/src/sumcheck/verifier.rs:14-113
//
// The transcript is the caller's (Monolith width 12, rate 8): the proof continues
// it, as `prove(.., transcript)` does in the reference, so the layers above (an
// einsum block, a fold-tree node) keep one transcript across their sumchecks.
#include <vector>
#include "../agl_traits.cuh"
#include "linear_sumcheck_state.cuh"
#include "agl_transcript.hpp"

using namespace mb;
using namespace mb::sc;

namespace mbhost {

using AglSumcheckStateExt2 = LinearSumcheckState<AglBase, AglExt2>;
using AglTranscript = aglm::Transcript;

static const uint8_t L_NUM_VAR[] = "num_var", L_NUM_POLY[] = "num_poly", L_MSG[] = "round_message",
                     L_CHALLENGE[] = "challenge";

static Ext2 aext2_mul_host(Ext2 a, Ext2 b) {
    agl::E2 r = agl::e2_canon(agl::e2_mul(agl::E2{a.c0, a.c1}, agl::E2{b.c0, b.c1}));
    return Ext2{r.c0, r.c1};
}
static Ext2 aext2_add_host(Ext2 a, Ext2 b) {
    return Ext2{agl::canon(agl::add(a.c0, b.c0)), agl::canon(agl::add(a.c1, b.c1))};
}
static Ext2 challenge_ext2(AglTranscript& t) {
    uint64_t w[2];
    t.challenge_vector(L_CHALLENGE, sizeof(L_CHALLENGE) - 1, w, 2);  // label once, two squeezes (transcript.rs:120-125)
    return Ext2{w[0], w[1]};
}

static int prove_linear(const uint64_t* d_tables, int d, int num_var, bool base_field, AglTranscript& t,
                        uint64_t* round_msgs, uint64_t* challenges, uint64_t* final_evals, uint64_t* final_eval) {
    t.append_u64(L_NUM_VAR, sizeof(L_NUM_VAR) - 1, (uint64_t)num_var);
    t.append_u64(L_NUM_POLY, sizeof(L_NUM_POLY) - 1, (uint64_t)d);
    AglSumcheckStateExt2 st;
    int rc = st.init_device(d_tables, d, num_var, base_field);
    if (rc != MB_OK) return rc;
    std::vector<Ext2> msg;
    bool label_absorbed = false;   // the first label of a round goes in while the round's kernel runs
    for (int round = 0; round < num_var; round++) {
        rc = st.compute_round_message(msg);
        if (rc != MB_OK) return rc;
        for (int c = 0; c <= d; c++) {
            if (c > 0 || !label_absorbed) t.begin_append(L_MSG, sizeof(L_MSG) - 1);
            t.finish_append_ext2(msg[c].c0, msg[c].c1);
            round_msgs[((size_t)round * (d + 1) + c) * 2] = msg[c].c0;
            round_msgs[((size_t)round * (d + 1) + c) * 2 + 1] = msg[c].c1;
        }
        Ext2 r = challenge_ext2(t);
        if (challenges) {
            challenges[2 * round] = r.c0;
            challenges[2 * round + 1] = r.c1;
        }
        rc = st.fold(r);
        if (rc != MB_OK) return rc;
        label_absorbed = round + 1 < num_var;
        if (label_absorbed) t.begin_append(L_MSG, sizeof(L_MSG) - 1);
    }
    std::vector<Ext2> fe;
    rc = st.final_evaluations(fe);
    if (rc != MB_OK) return rc;
    Ext2 prod{1, 0};
    for (int i = 0; i < d; i++) {
        if (final_evals) {
            final_evals[2 * i] = fe[i].c0;
            final_evals[2 * i + 1] = fe[i].c1;
        }
        prod = aext2_mul_host(prod, fe[i]);
    }
    final_eval[0] = prod.c0;
    final_eval[1] = prod.c1;
    return MB_OK;
}

// The same protocol for the three tables a, b, eq(t, x) (extended by copies over the variables from eq_vars on; a
// table of ones when eq_vars is 0) without forming the third: several rounds per pass (pair_sumcheck.cuh). base: a and
// b are base field words. Messages are those of the three-table prover, P(0..3).
int prove_pair_with_eq(const uint64_t* d_a, const uint64_t* d_b, bool base, int num_var, const uint64_t* eq_pt, int eq_vars,
                       AglTranscript& t, uint64_t* round_msgs, uint64_t* challenges, uint64_t* final_evals, uint64_t* final_eval) {
    using Pair = PairSumcheck<pr::AglF, PairAgl>;
    using H = Pair::H;
    using E2 = agl::E2;
    Pair st;
    int rc = st.init(d_a, d_b, 0, 1, num_var, base, eq_pt, eq_vars);
    if (rc != MB_OK) return rc;
    t.append_u64(L_NUM_VAR, sizeof(L_NUM_VAR) - 1, (uint64_t)num_var);
    t.append_u64(L_NUM_POLY, sizeof(L_NUM_POLY) - 1, 3);
    for (int round = 0; round < num_var; round++) {
        t.begin_append(L_MSG, sizeof(L_MSG) - 1);   // the first label goes in while a pass runs
        E2 t0, t1, t2;
        rc = st.sums(t0, t1, t2);
        if (rc != MB_OK) return rc;
        const E2 s12 = H::add(t1, t2), p2 = H::sub(H::add(s12, s12), t0);                        // 2 t1 + 2 t2 - t0
        const E2 t22 = H::add(t2, t2), p3 = H::add(H::sub(H::add(p2, t1), t0), H::add(t22, t22));   // 3 t1 + 6 t2 - 2 t0
        E2 msg[4] = {t0, t1, p2, p3};
        if (eq_vars > 0) {
            E2 lam = st.eq_scale(), step{0, 0};
            if (round < eq_vars) {
                const E2 c = st.eq_coord(round), one{1, 0};
                step = H::mul(lam, H::sub(H::add(c, c), one));
                lam = H::mul(lam, H::sub(one, c));
            }
            for (int c = 0; c < 4; c++) {
                msg[c] = H::mul(lam, msg[c]);
                lam = H::add(lam, step);
            }
        }
        for (int c = 0; c < 4; c++) {
            if (c > 0) t.begin_append(L_MSG, sizeof(L_MSG) - 1);
            t.finish_append_ext2(msg[c].c0, msg[c].c1);
            round_msgs[((size_t)round * 4 + c) * 2] = msg[c].c0;
            round_msgs[((size_t)round * 4 + c) * 2 + 1] = msg[c].c1;
        }
        const Ext2 r = challenge_ext2(t);
        if (challenges) {
            challenges[2 * round] = r.c0;
            challenges[2 * round + 1] = r.c1;
        }
        rc = st.fold(E2{r.c0, r.c1});
        if (rc != MB_OK) return rc;
    }
    E2 f[3];
    rc = st.finals(&f[0], &f[1]);
    if (rc != MB_OK) return rc;
    f[2] = st.eq_scale();
    for (int i = 0; i < 3 && final_evals; i++) {
        final_evals[2 * i] = f[i].c0;
        final_evals[2 * i + 1] = f[i].c1;
    }
    const E2 prod = H::mul(H::mul(f[0], f[1]), f[2]);
    final_eval[0] = prod.c0;
    final_eval[1] = prod.c1;
    return MB_OK;
}

// Lagrange interpolation through x = 0..n-1, evaluated at x (verifier.rs:91-113).
// The denominators are products of small integers: their inverses are formed once per node count.
static Ext2 interpolate_and_evaluate(const Ext2* evals, int n, Ext2 x) {
    using H = PairHost<pr::AglF, PairAgl>;
    using E2 = agl::E2;
    struct Table {
        uint64_t inv[MAX_D + 2][MAX_D + 1];
        Table() {
            for (int m = 1; m <= MAX_D + 1; m++)
                for (int i = 0; i < m; i++) {
                    uint64_t den = 1;
                    for (int j = 0; j < m; j++)
                        if (j != i) den = agl::mul(den, agl::sub((uint64_t)i, (uint64_t)j));
                    inv[m][i] = agl::canon(agl::inv(den));
                }
        }
    };
    static const Table table;
    // prefix and suffix products of x - j
    E2 d[MAX_D + 1], pre[MAX_D + 2], suf[MAX_D + 2];
    pre[0] = suf[n] = E2{1, 0};
    for (int j = 0; j < n; j++) d[j] = H::sub(E2{x.c0, x.c1}, E2{(uint64_t)j, 0});
    for (int j = 0; j < n; j++) pre[j + 1] = H::mul(pre[j], d[j]);
    for (int j = n - 1; j >= 0; j--) suf[j] = H::mul(suf[j + 1], d[j]);
    typename H::Dot sum;
    for (int i = 0; i < n; i++) {
        const E2 e{evals[i].c0, evals[i].c1};
        const uint64_t w = table.inv[n][i];
        sum.mac(E2{PairAgl::canon(PairAgl::red((hf::u128)e.c0 * w)), PairAgl::canon(PairAgl::red((hf::u128)e.c1 * w))}, H::mul(pre[i], suf[i + 1]));
    }
    const E2 r = sum.value();
    return Ext2{r.c0, r.c1};
}

}  // namespace mbhost

extern "C" {

// Whole sumcheck proof for d tables of 2^num_var elements already on the device
// (poly-major; base_field != 0: one word per element, else (c0, c1)). `transcript`
// is a handle from agl_transcript_create and is advanced by the proof. Host outputs:
// round_msgs[num_var][d+1][2], challenges[num_var][2] (may be NULL),
// final_evals[d][2] (may be NULL), final_eval[2] = product of the final evaluations.
int agl_sumcheck_prove_device_ffi(const uint64_t* d_tables, int d, int num_var, int base_field, void* transcript,
                                  uint64_t* round_msgs, uint64_t* challenges, uint64_t* final_evals,
                                  uint64_t* final_eval) {
    if (!transcript || !round_msgs || !final_eval) return MB_ERR_ARG;
    return mbhost::prove_linear(d_tables, d, num_var, base_field != 0, *static_cast<mbhost::AglTranscript*>(transcript),
                                round_msgs, challenges, final_evals, final_eval);
}

// Same proof from host tables: uploads them, proves, frees the device copy.
int agl_sumcheck_prove_host_ffi(const uint64_t* h_tables, int d, int num_var, int base_field, void* transcript,
                                uint64_t* round_msgs, uint64_t* challenges, uint64_t* final_evals,
                                uint64_t* final_eval) {
    if (d < 1 || d > MAX_D || num_var < 0 || num_var > 40 || !h_tables) return MB_ERR_ARG;
    size_t words = ((size_t)1 << num_var) * (size_t)d * (base_field ? 1 : 2);
    uint64_t* d_tables = nullptr;
    MB_CUDA(pool_alloc((void**)&d_tables, words * sizeof(uint64_t)));
    int rc = MB_OK;
    if (cudaMemcpyAsync(d_tables, h_tables, words * sizeof(uint64_t), cudaMemcpyHostToDevice, MB_STREAM) != cudaSuccess)
        rc = MB_ERR_CUDA;
    if (rc == MB_OK)
        rc = agl_sumcheck_prove_device_ffi(d_tables, d, num_var, base_field, transcript, round_msgs, challenges,
                                           final_evals, final_eval);
    pool_free(d_tables);
    return rc;
}

// SumcheckVerifier::verify on the host: *ok = 1 when every round's P(0) + P(1)
// equals the running claim and the last claim equals final_eval; the challenges
// (num_var pairs) are written when `challenges` is not NULL. The transcript is
// advanced exactly as the prover's, up to the round that fails.
int agl_sumcheck_verify_ffi(const uint64_t* round_msgs, const uint64_t* final_eval, const uint64_t* claimed_sum, int d,
                            int num_var, void* transcript, uint64_t* challenges, int* ok) {
    using namespace mbhost;
    if (!transcript || !ok || !final_eval || !claimed_sum || d < 1 || d > MAX_D || num_var < 0 || (num_var && !round_msgs))
        return MB_ERR_ARG;
    AglTranscript& t = *static_cast<AglTranscript*>(transcript);
    *ok = 0;
    t.append_u64(L_NUM_VAR, sizeof(L_NUM_VAR) - 1, (uint64_t)num_var);
    t.append_u64(L_NUM_POLY, sizeof(L_NUM_POLY) - 1, (uint64_t)d);
    Ext2 current{agl::canon(claimed_sum[0]), agl::canon(claimed_sum[1])};
    std::vector<Ext2> msg(d + 1);
    for (int round = 0; round < num_var; round++) {
        for (int c = 0; c <= d; c++) {
            const uint64_t* w = round_msgs + ((size_t)round * (d + 1) + c) * 2;
            msg[c] = Ext2{agl::canon(w[0]), agl::canon(w[1])};
        }
        Ext2 sum = aext2_add_host(msg[0], msg[1]);
        if (sum.c0 != current.c0 || sum.c1 != current.c1) return MB_OK;
        for (int c = 0; c <= d; c++) t.append_ext2(L_MSG, sizeof(L_MSG) - 1, msg[c].c0, msg[c].c1);
        Ext2 r = challenge_ext2(t);
        if (challenges) {
            challenges[2 * round] = r.c0;
            challenges[2 * round + 1] = r.c1;
        }
        current = interpolate_and_evaluate(msg.data(), d + 1, r);
    }
    *ok = current.c0 == agl::canon(final_eval[0]) && current.c1 == agl::canon(final_eval[1]);
    return MB_OK;
}

}  // extern "C"
