// Host layer above the C-ABI for Basefold over Goldilocks: folding table,
// commitment and extension-field opening, written in C++ where the reference has
// Rust (no Rust toolchain on the build machine).
//
//   BasefoldTable        goldilocks-cuda-rs/src/basefold.rs:267-362
//   DeviceMerkleTree     goldilocks-cuda-rs/src/merkle.rs:20-160
//   BasefoldCommitment   goldilocks-cuda-rs/src/basefold.rs:368-414 (commit_device)
//   open_ext2            goldilocks-cuda-rs/src/basefold.rs:578-863
//   extract_ext2_queries goldilocks-cuda-rs/src/basefold.rs:2310-2402
//
// The protocol order, every transcript interaction and every value that enters
// the proof are the reference's. The work between them is organised for the
// B200: the claimed value is read off the first oracle (eval = p(0) + p(1), one
// pass fewer), the inner sumcheck runs several rounds per pass over the
// bit-reversed evaluations (OpenSumcheck), the codeword is folded by the kernels
// that hash its leaves, each round issues them back to back and waits
// once, the last few rounds are folded and hashed by the host (host_leaves),
// and the query phase is one gather kernel and one copy.
#include "gl_basefold_common.cuh"

namespace mbhost {

// out[i], i < n: the codeword `in` folded on r (entries: its table level)
static void fold_on_host(const uint64_t* in, const uint64_t* entries, gl::E2 r, uint64_t* out, size_t n) {
    const uint64_t r1w = gl::mul_small(r.c1, 7);
    for (size_t i = 0; i < n; i++) {
        const gl::E2 e = bf::fold_pair_ext(gl::E2{in[4 * i], in[4 * i + 1]}, gl::E2{in[4 * i + 2], in[4 * i + 3]},
                                           make_ulonglong2(entries[2 * i], entries[2 * i + 1]), r, r1w);
        out[2 * i] = e.c0;
        out[2 * i + 1] = e.c1;
    }
}

// Of an opening's scratch block: sums of the inner sumcheck from word 0, a tree's last device layer from NODE_WORD, the queries' indices.
constexpr size_t NODE_WORD = 64, QUERY_WORD = 1024;
static_assert((size_t)2 << pr::MAX_B <= NODE_WORD && NODE_WORD + 4 * HOST_TOP <= QUERY_WORD && QUERY_WORD < ScratchPool::WORDS, "one after another");

// open_ext2 (basefold.rs:578-863). Writes the proof as
//   eval[2] | oracles[nv][3][2] | folded_roots[nv-1][4] | final_codeword[2^lr][2] |
//   per query: index, nv value pairs [2][2], path in the commitment tree,
//   paths in the nv-1 folded trees (sibling digests bottom-up).
int open_ext2(const BasefoldCommitment& cm, const uint64_t* point, const BasefoldTable& table, Transcript& t,
              int num_queries, uint64_t* proof) {
    const int nv = cm.num_vars, lr = cm.log_rate;
    if (nv < 2 || nv > 38 || table.num_vars != nv || table.log_rate != lr || table.rounds < nv || num_queries < 0)
        return MB_ERR_ARG;
    const size_t n = (size_t)1 << nv, cw_len = (size_t)1 << (nv + lr);
    uint64_t* p_eval = proof;
    uint64_t* p_oracles = proof + 2;
    uint64_t* p_roots = p_oracles + (size_t)nv * 6;
    uint64_t* p_final = p_roots + (size_t)(nv - 1) * 4;
    uint64_t* p_queries = p_final + ((size_t)2 << lr);

    ScopedScratch pin;
    // The first round of the host's own: its codeword is folded, and hashed, from a copy of the one before. (Never round 0; nv - 1: none.)
    const auto leaves_of = [&](int round) { return cw_len >> (round + 2); };
    int host_round = 1;
    while (host_round < nv - 1 && leaves_of(host_round) > host_leaves(cm.hash)) host_round++;
    const bool on_host = host_round < nv - 1;
    const size_t copy_words = on_host ? 8 * leaves_of(host_round) : 0;
    // host-hashed tree tops on their way up; the copy; the host's rounds: by round the codeword (a pair of elements a leaf), the tree
    std::vector<size_t> own(nv, 0);
    size_t own_words = 0;
    for (int i = host_round; i < nv - 1; i++) {
        own[i] = own_words;
        own_words += 4 * leaves_of(i) + 4 * (2 * leaves_of(i) - 1);
    }
    const size_t staging_words = 4 * (HOST_TOP - 1) * (size_t)nv;
    uint64_t* top_staging = pinned_arena(staging_words + copy_words + own_words);
    if (!pin.p || !top_staging) return MB_ERR_CUDA;
    uint64_t *copied = top_staging + staging_words, *host_rounds = copied + copy_words;
    uint64_t* nodes = pin.p + NODE_WORD;
    OpenSumcheck sc;
    int rc = sc.init(cm.d_bh_evals.p, nv, point, pin.p, pin.b.dev);
    if (rc != MB_OK) return rc;
    t.observe_hash(cm.root);   // while the first pass runs
    for (int i = 0; i < nv; i++) t.observe_ext2(Ext2{point[2 * i], point[2 * i + 1]});
    rc = sc.wait();
    if (rc != MB_OK) return rc;
    // oracle 0 and the claimed value eval = p(0) + p(1) = 2 c0 + c1 + c2
    sc.oracle(p_oracles);
    {
        gl::E2 c0{p_oracles[0], p_oracles[1]}, c1{p_oracles[2], p_oracles[3]}, c2{p_oracles[4], p_oracles[5]};
        gl::E2 ev = gl::e2_canon(gl::e2_add(gl::e2_add(c0, c0), gl::e2_add(c1, c2)));
        p_eval[0] = ev.c0;
        p_eval[1] = ev.c1;
    }
    for (int k = 0; k < 3; k++) t.observe_ext2(Ext2{p_oracles[2 * k], p_oracles[2 * k + 1]});

    // folded codewords and trees, kept for the query phase
    std::vector<std::unique_ptr<DevBuf>> fcw(nv), ftree(nv - 1);
    {
        size_t len = cw_len / 2;
        for (int i = 0; i < (on_host ? host_round : nv); i++) {
            fcw[i].reset(new DevBuf);
            rc = fcw[i]->alloc(2 * len);
            if (rc != MB_OK) return rc;
            if (i < nv - 1) {
                ftree[i].reset(new DevBuf);
                rc = ftree[i]->alloc(4 * (len - 1 > 0 ? len - 1 : 1));
                if (rc != MB_OK) return rc;
            }
            len /= 2;
        }
    }

    size_t cw_pairs = cw_len / 2;
    for (int round = 0; round < nv - 1; round++) {
        Ext2 ch = t.sample_challenge_ext2();
        gl::E2 r{ch.c0, ch.c1};
        // kernels write their results straight into pinned host memory: a round is its launches and one wait for them, no copy
        // command
        rc = sc.fold(r);
        if (rc != MB_OK) return rc;
        uint64_t* po = p_oracles + 6 * (size_t)(round + 1);
        uint64_t* root = p_roots + 4 * (size_t)round;
        if (round >= host_round) {   // beside a pass of the inner sumcheck, if the fold queued one
            if (round == host_round) rc = await_words(copied, copy_words);
            if (rc != MB_OK) return rc;
            const size_t n_leaves = leaves_of(round);
            uint64_t *cw = host_rounds + own[round], *tree = cw + 4 * n_leaves;
            fold_on_host(round == host_round ? copied : host_rounds + own[round - 1], table.host_level(round), r, cw, 2 * n_leaves);
            static const uint64_t none[4] = {0, 0, 0, 0};
            for (size_t k = 0; k < n_leaves; k++) std::memcpy(tree + 4 * k, host_compress(cm.hash, cw + 4 * k, none).w, 32);
            host_hash_top(cm.hash, tree, n_leaves, tree + 4 * n_leaves, root);
            rc = sc.wait();
            if (rc != MB_OK) return rc;
            sc.oracle(po);
            for (int k = 0; k < 3; k++) t.observe_ext2(Ext2{po[2 * k], po[2 * k + 1]});
            t.observe_hash(root);
            cw_pairs /= 2;
            continue;
        }
        // codeword fold with this round's table level, and its tree up to the layer the host takes over
        const size_t leaves = cw_pairs / 2;
        const mk::FoldSource f{round == 0 ? cm.d_codeword.p : fcw[round - 1]->p, table.device_level_ptr(round), fcw[round]->p, r};
        const size_t top = host_top(cm.hash), top_nodes = leaves < top ? leaves : top;
        expect_words(nodes, 4 * top_nodes);
        rc = queue_fold_tree(cm.hash, round == 0, f, ftree[round]->p, leaves, nodes);
        if (rc == MB_OK && round + 1 == host_round && on_host) {
            expect_words(copied, copy_words);
            MB_KERNEL_ON("send_tables", MB_STREAM);
            pr::send_tables_kernel<pr::GlF><<<1, pr::BLK, 0, MB_STREAM>>>(fcw[round]->p, nullptr, 0, copy_words, copied);
            if (cudaGetLastError() != cudaSuccess) rc = MB_ERR_CUDA;
        }
        if (rc == MB_OK) rc = await_words(nodes, 4 * top_nodes);
        if (rc == MB_OK) rc = sc.wait();
        if (rc != MB_OK) return rc;
        sc.oracle(po);
        rc = host_finish_top(cm.hash, nodes, top_nodes, top_staging + 4 * (HOST_TOP - 1) * (size_t)round,
                             ftree[round]->p, leaves, root, MB_STREAM);
        if (rc != MB_OK) return rc;
        for (int k = 0; k < 3; k++) t.observe_ext2(Ext2{po[2 * k], po[2 * k + 1]});
        t.observe_hash(root);
        cw_pairs /= 2;
    }

    // last challenge: final fold, no tree
    {
        Ext2 ch = t.sample_challenge_ext2();
        gl::E2 r{ch.c0, ch.c1};
        if (on_host) {
            fold_on_host(host_rounds + own[nv - 2], table.host_level(nv - 1), r, p_final, cw_pairs);
        } else {
            MB_KERNEL_ON("fold_ext2", MB_STREAM);
            bf::fold_ext2_kernel<<<grid_for(cw_pairs, 256, 8), 256, 0, MB_STREAM>>>(
                fcw[nv - 2]->p, table.device_level_ptr(nv - 1), r, fcw[nv - 1]->p, cw_pairs);
        }
        if (cudaGetLastError() != cudaSuccess) return MB_ERR_CUDA;
        if (!on_host)
            MB_CUDA(cudaMemcpyAsync(p_final, fcw[nv - 1]->p, sizeof(uint64_t) * ((size_t)2 << lr), cudaMemcpyDeviceToHost, MB_STREAM));
    }

    // queries: all indices first (basefold.rs:2321-2326), then one gather
    if (num_queries > 0) {
        // the kernel reads the indices where the host leaves them, as far as there is room
        uint64_t* host_idx = pin.p + QUERY_WORD;
        const bool direct = num_queries <= (int)(ScratchPool::WORDS - QUERY_WORD);
        std::vector<uint64_t> idx(direct ? 0 : num_queries);
        if (!direct) host_idx = idx.data();
        for (int q = 0; q < num_queries; q++) host_idx[q] = t.sample_challenge() % (uint64_t)(cw_len / 2);
        size_t qw = query_words(nv, lr);
        DevBuf d_idx, d_q, d_own;   // d_own: the host's rounds
        rc = direct ? MB_OK : d_idx.alloc(num_queries);
        if (rc == MB_OK) rc = d_q.alloc(qw * num_queries);
        if (rc != MB_OK) return rc;
        if (!direct) MB_CUDA(cudaMemcpyAsync(d_idx.p, idx.data(), sizeof(uint64_t) * num_queries, cudaMemcpyHostToDevice, MB_STREAM));
        QueryLevels lv;
        lv.nv = nv; lv.lr = lr;
        lv.commit_cw = cm.d_codeword.p;
        lv.commit_tree = cm.d_tree.p;
        if (on_host) {
            rc = d_own.alloc(own_words);
            if (rc != MB_OK) return rc;
            MB_CUDA(cudaMemcpyAsync(d_own.p, host_rounds, sizeof(uint64_t) * own_words, cudaMemcpyHostToDevice, MB_STREAM));
        }
        for (int i = 0; i <= nv - 2; i++) {
            lv.fcw[i] = i < host_round ? fcw[i]->p : d_own.p + own[i];
            lv.ftree[i] = i < host_round ? ftree[i]->p : d_own.p + own[i] + 4 * leaves_of(i);
        }
        {
            MB_KERNEL_ON("query_gather", MB_STREAM);
            query_gather_kernel<<<num_queries, 128, 0, MB_STREAM>>>(lv, direct ? host_idx : d_idx.p, d_q.p, qw);
        }
        if (cudaGetLastError() != cudaSuccess) return MB_ERR_CUDA;
        MB_CUDA(cudaMemcpyAsync(p_queries, d_q.p, sizeof(uint64_t) * qw * num_queries, cudaMemcpyDeviceToHost, MB_STREAM));
        MB_CUDA(cudaStreamSynchronize(MB_STREAM));
    } else {
        MB_CUDA(cudaStreamSynchronize(MB_STREAM));
    }
    return MB_OK;
}

// Evaluations on the device, or in host memory.
static int commit(const uint64_t* d_evals, const uint64_t* h_evals, int nv, int lr, void** commitment, uint64_t* h_root) {
    if (!commitment || (!d_evals && !h_evals)) return MB_ERR_ARG;
    auto c = std::make_unique<BasefoldCommitment>();
    int rc = c->allocate(nv, lr);
    if (rc != MB_OK) return rc;
    DevBuf uploaded;
    if (h_evals) {
        rc = uploaded.alloc((size_t)1 << nv);
        if (rc != MB_OK) return rc;
        MB_CUDA(cudaMemcpyAsync(uploaded.p, h_evals, sizeof(uint64_t) << nv, cudaMemcpyHostToDevice, MB_STREAM));
        d_evals = uploaded.p;
    }
    rc = c->commit_device(d_evals);
    if (rc != MB_OK) return rc;
    if (h_root) std::memcpy(h_root, c->root, 32);
    *commitment = c.release();
    return MB_OK;
}

}  // namespace mbhost

// ---- C-ABI of the host layer -----------------------------------------------------------
using mbhost::BasefoldCommitment;
using mbhost::BasefoldTable;

extern "C" {

// Selects the Merkle hash of later commitments: 0 Poseidon2 (default), 1 Monolith.
int basefold_set_merkle_hash(int hash) {
    if (hash != 0 && hash != 1) return MB_ERR_ARG;
    mbhost::g_merkle_hash.store(hash);
    return MB_OK;
}

size_t basefold_proof_words(int num_vars, int log_rate, int num_queries) {
    return mbhost::proof_words(num_vars, log_rate, num_queries);
}

int basefold_table_create(int num_vars, int log_rate, int num_rounds, uint64_t seed, void** table) {
    if (!table) return MB_ERR_ARG;
    auto* t = new BasefoldTable;
    int rc = t->generate(num_vars, log_rate, num_rounds, seed);
    if (rc != MB_OK) { delete t; return rc; }
    *table = t;
    return MB_OK;
}
int basefold_table_destroy(void* table) { delete static_cast<BasefoldTable*>(table); return MB_OK; }
size_t basefold_table_entries(const void* table) { return static_cast<const BasefoldTable*>(table)->entries; }
// (point, weight) pairs, levels back to back, to host memory.
int basefold_table_download(const void* table, uint64_t* h_entries) {
    auto* t = static_cast<const BasefoldTable*>(table);
    MB_CUDA(cudaMemcpyAsync(h_entries, t->d_entries.p, t->entries * 16, cudaMemcpyDeviceToHost, MB_STREAM));
    return cudaStreamSynchronize(MB_STREAM) == cudaSuccess ? MB_OK : MB_ERR_CUDA;
}
const uint64_t* basefold_table_level_ptr(const void* table, int level) {
    return static_cast<const BasefoldTable*>(table)->device_level_ptr(level);
}

int basefold_commit_device(const uint64_t* d_evals, int num_vars, int log_rate, void** commitment, uint64_t* h_root) {
    return mbhost::commit(d_evals, nullptr, num_vars, log_rate, commitment, h_root);
}
int basefold_commit_host(const uint64_t* h_evals, int num_vars, int log_rate, void** commitment, uint64_t* h_root) {
    return mbhost::commit(nullptr, h_evals, num_vars, log_rate, commitment, h_root);
}
int basefold_commitment_destroy(void* commitment) { delete static_cast<BasefoldCommitment*>(commitment); return MB_OK; }
// Device pointers of the commitment's parts (owned by the commitment).
const uint64_t* basefold_commitment_codeword(const void* c) { return static_cast<const BasefoldCommitment*>(c)->d_codeword.p; }
const uint64_t* basefold_commitment_bh_evals(const void* c) { return static_cast<const BasefoldCommitment*>(c)->d_bh_evals.p; }
const uint64_t* basefold_commitment_tree(const void* c) { return static_cast<const BasefoldCommitment*>(c)->d_tree.p; }

// Opening at an extension-field point (h_point: num_vars (c0, c1) pairs) with
// the transcript started as Transcript::new(label). h_proof must hold
// basefold_proof_words(...) words; h_transcript_state (8 words) may be NULL.
int basefold_open_ext2(const void* commitment, const uint64_t* h_point, const void* table, const uint8_t* label,
                       size_t label_len, int num_queries, uint64_t* h_proof, uint64_t* h_transcript_state) {
    if (!commitment || !h_point || !table || !h_proof) return MB_ERR_ARG;
    mbhost::Transcript t(label, label_len);
    int rc = mbhost::open_ext2(*static_cast<const BasefoldCommitment*>(commitment), h_point,
                               *static_cast<const BasefoldTable*>(table), t, num_queries, h_proof);
    if (rc == MB_OK && h_transcript_state) std::memcpy(h_transcript_state, t.state(), 64);
    return rc;
}

// Commit + open from host evaluations in one call; the commitment is dropped
// afterwards. h_root receives the commitment root.
int basefold_prove_host(const uint64_t* h_evals, int num_vars, int log_rate, const uint64_t* h_point, const void* table,
                        const uint8_t* label, size_t label_len, int num_queries, uint64_t* h_root, uint64_t* h_proof) {
    void* c = nullptr;
    int rc = basefold_commit_host(h_evals, num_vars, log_rate, &c, h_root);
    if (rc != MB_OK) return rc;
    rc = basefold_open_ext2(c, h_point, table, label, label_len, num_queries, h_proof, nullptr);
    basefold_commitment_destroy(c);
    return rc;
}

}  // extern "C"
