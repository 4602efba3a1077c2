"""The sizes at which a prover changes kernels: tables that go to the host, several rounds per pass, one round per pass,
uneven last blocks; hashing layers around the switch between lanes and threads; column chunks of the tensor-core commit.
Bit equality with the CPU oracle."""
import ctypes

import numpy as np
import pytest

from matrix_b200.ffi import DeviceBuffer, load_agl, load_gl
from matrix_b200.inputs import AGL_Q, GL_P, field_elems, splitmix64
from oracle import pyoracle

from .test_agl_sumcheck_prover_gpu import _prove, _state, _transcript
from .test_ajtai_gpu import KEY
from .test_basefold_gpu import test_commit_open_matches_oracle as basefold_matches_oracle
from .test_batched_gpu import test_whole_proof_inside_the_library as batched_matches_oracle
from .test_monolith_gpu import test_commit_open_with_monolith_trees as monolith_basefold_matches_oracle
from .test_sumcheck_gpu import test_whole_proof_matches_oracle as gl_sumcheck_matches_oracle

pytestmark = pytest.mark.gpu

# one table: host up to 2^8, then four rounds a pass; two: host up to 2^10 (base) or 2^9, blocks of 4 and 3 rounds, on the
# tensor cores from 2^14; three: passes from 2^9, on the tensor cores from 2^15; four: to 2^13
ROUNDS = [(2, 13), (2, 14), (2, 15), (2, 16), (3, 19), (1, 8), (1, 9), (1, 13), (1, 17), (2, 1), (2, 9), (2, 10), (2, 11), (2, 18), (2, 19), (3, 8), (3, 9), (3, 14), (3, 15),
          (3, 16), (3, 17), (3, 18), (4, 8), (4, 10), (4, 13), (4, 14), (4, 16)]


@pytest.fixture(scope="module")
def gl():
    lib = load_gl()
    assert lib.goldilocks_cuda_init() == 0
    assert lib.monolith_cuda_init() == 0
    return lib


@pytest.mark.parametrize("d,nv", ROUNDS)
@pytest.mark.parametrize("base", [True, False])
def test_sumcheck_rounds_agl(d, nv, base):
    lib = load_agl()
    raw = splitmix64(900 + 100 * d + nv, (d << nv) * (1 if base else 2))   # words at or above q among them
    raw[:3] = [AGL_Q, 2**64 - 1, AGL_Q - 1][:len(raw[:3])]
    want = pyoracle.agl_sumcheck_prove(raw, d, nv, base, b"edges")
    h = _transcript(lib, b"edges")
    got = _prove(lib, raw, d, nv, base, h)
    for g, w in zip(got + (_state(lib, h),), want):
        assert np.array_equal(g, np.array(w, dtype=np.uint64))
    lib.agl_transcript_destroy(h)


@pytest.mark.parametrize("d,nv", ROUNDS)
@pytest.mark.parametrize("base", [True, False])
def test_sumcheck_rounds_gl(gl, d, nv, base):
    gl_sumcheck_matches_oracle(gl, nv, d, base)


# passes that fold a few tiles, several threads an element: one to eight of them, whole tiles and parts, below, at and above 64 tiles of 256
# elements over the instances
@pytest.mark.parametrize("K,nv", [(1, 11), (1, 12), (1, 17), (2, 10), (3, 13), (7, 12), (16, 10), (16, 14), (24, 9), (31, 12), (33, 13), (64, 11)])
def test_small_folds(K, nv):
    batched_matches_oracle(K, nv, 0)


# three and four tables by tiles of 16 elements: from four clusters of eight blocks on (2^9 elements), and folds of two, three and no challenges
@pytest.mark.parametrize("d,nv", [(3, 9), (3, 10), (3, 11), (3, 12), (3, 13), (4, 9), (4, 11), (4, 12), (4, 15)])
@pytest.mark.parametrize("base", [True, False])
def test_small_products(gl, d, nv, base):
    gl_sumcheck_matches_oracle(gl, nv, d, base)
    test_sumcheck_rounds_agl(d, nv, base)


@pytest.mark.parametrize("d", [6, 7, 8])
@pytest.mark.parametrize("blocks", [1, 148, 149, 600])   # a block per SM, and more
def test_many_tables(gl, oracle, d, blocks):
    n = 1 << 15
    tabs, r = field_elems(950 + d, 2 * n * d), [2**63 + 11, 5]
    d_in, d_out, d_part = DeviceBuffer.from_numpy(gl, tabs), DeviceBuffer(gl, tabs.nbytes), DeviceBuffer(gl, blocks * (d + 1) * 16)

    def totals():
        return [sum(int(x) for x in col) % GL_P for col in d_part.to_numpy().reshape(blocks, -1).T]

    want, folded = np.zeros(2 * (d + 1), dtype=np.uint64), tabs.copy()
    oracle.oracle_gl_round_message_ext2(tabs.ctypes.data, d, n, n // 2, want.ctypes.data)
    assert gl.sumcheck_round_message_ext2_ffi(d_in.ptr, d_part.ptr, d, n, n // 2, blocks) == 0
    assert totals() == [int(x) for x in want]
    oracle.oracle_gl_fold_ext2(tabs.ctypes.data, folded.ctypes.data, *r, d, n, n // 2)
    oracle.oracle_gl_round_message_ext2(folded.ctypes.data, d, n, n // 4, want.ctypes.data)
    assert gl.sumcheck_fold_round_ext2_ffi(d_in.ptr, d_out.ptr, *r, d, n, n // 4, d_part.ptr, blocks) == 0
    assert totals() == [int(x) for x in want]
    got = d_out.to_numpy().reshape(d, 2 * n)[:, :n]
    assert np.array_equal(got, folded.reshape(d, 2 * n)[:, :n])


@pytest.mark.parametrize("K,nv", [(1, 9), (2, 9), (3, 10), (4, 12), (7, 13), (64, 4), (64, 11), (1, 18), (5, 17),
                                  (1, 13), (1, 14), (1, 20), (3, 13), (16, 11), (16, 14), (64, 8), (64, 10)])
def test_batched_rounds(K, nv):
    batched_matches_oracle(K, nv, 0)


@pytest.mark.parametrize("nv,lr,nq", [(2, 2, 1), (2, 3, 2), (5, 2, 3), (8, 3, 7), (9, 0, 4), (11, 1, 8), (12, 2, 8), (14, 1, 8), (15, 2, 8)])
def test_basefold_sizes(gl, nv, lr, nq):
    basefold_matches_oracle(gl, nv, lr, nq)
    monolith_basefold_matches_oracle(gl, nv, lr, nq)


@pytest.mark.parametrize("nv,lr,nq", [(3, 0, 2), (4, 4, 3), (4, 5, 3), (3, 6, 2), (6, 1, 0), (9, 1, 12)])
def test_basefold_rounds_of_the_host(gl, nv, lr, nq):
    """The host folds and hashes the rounds of few leaves: one round, several, none, in either hash."""
    basefold_matches_oracle(gl, nv, lr, nq)
    if nq:   # (the other test ends with openings that the wrong hash must not verify)
        monolith_basefold_matches_oracle(gl, nv, lr, nq)


@pytest.mark.parametrize("nq", [7168, 7169])
def test_basefold_queries_beyond_the_scratch_block(gl, nq):
    """Up to 7168 query indices are read where the host leaves them, more go up in a buffer."""
    basefold_matches_oracle(gl, 3, 1, nq)


def test_poseidon2_with_a_missed_carry(gl, oracle):
    """The throughput form adds without the rare carry and borrow repairs and redoes a permutation that needed one. The
    first round constant makes lane 0 of this state 2^48 before its S-box, whose square is a power of two that does;
    the extreme residues come along."""
    states = field_elems(77, 8 * 64)
    states[0] = (2**48 - 0xdd5743e7f2a5a5d9) % GL_P
    states[1:8] = 0
    states[8:16] = GL_P - 1
    states[16:24] = 2**32 - 1
    d_in, d_out = DeviceBuffer.from_numpy(gl, states), DeviceBuffer(gl, states.nbytes)
    assert gl.poseidon2_hash_batch_ffi(d_in.ptr, d_out.ptr, 64) == 0
    got = d_out.to_numpy().reshape(64, 8)
    for k in range(64):
        s = (ctypes.c_uint64 * 8)(*[int(x) for x in states[8 * k:8 * k + 8]])
        oracle.gl_poseidon2_permute(s)
        assert list(got[k]) == list(s), k


@pytest.mark.parametrize("leaves,ext", [((1 << 20) - 2**19, False), (1 << 20, False), (1 << 20, True), (1 << 21, False)])
def test_poseidon2_tiles(gl, oracle, leaves, ext):
    """Layers of 2^20 permutations and more go in tiles (the smaller tree has none, the largest one with two such layers):
    words at the ends of their range, and leaves whose reduction needs the exact form, among them."""
    width = 4 if ext else 2
    cw = field_elems(78, leaves * width).reshape(leaves, width)
    cw[3], cw[130] = GL_P - 1, 2**32 - 1
    for k in (5, 127, 128, leaves - 1):
        cw[k] = 0
        cw[k, 0] = (2**48 - 0xdd5743e7f2a5a5d9) % GL_P
    d_cw, d_t = DeviceBuffer.from_numpy(gl, cw.reshape(-1)), DeviceBuffer(gl, 32 * (2 * leaves - 1))
    assert (gl.poseidon2_merkle_tree_ext2_ffi if ext else gl.poseidon2_merkle_tree_gl_ffi)(d_cw.ptr, d_t.ptr, leaves) == 0
    exp = np.zeros(4 * (2 * leaves - 1), dtype=np.uint64)
    oracle.oracle_bf_merkle_tree(cw.ctypes.data, leaves, int(ext), exp.ctypes.data)
    assert np.array_equal(d_t.to_numpy(), exp)


# a layer of 2^15 permutations goes a thread each, 2^16 take three or four tiles an SM, 2^17 a second turn of some
@pytest.mark.parametrize("leaves,ext", [(1 << 15, True), (1 << 16, False), (1 << 16, True), (1 << 17, False)])
def test_poseidon2_tiles_of_few_turns(gl, oracle, leaves, ext):
    test_poseidon2_tiles(gl, oracle, leaves, ext)


@pytest.mark.parametrize("log_leaves", range(13))
@pytest.mark.parametrize("ext", [False, True])
def test_small_poseidon2_trees(gl, oracle, log_leaves, ext):
    """Eight lanes a permutation and a warp a permutation, by the number of levels left: every split of levels into launches, with
    leaves whose first product needs the exact form (2^96) in the lowest layer."""
    leaves, width = 1 << log_leaves, 4 if ext else 2
    cw = field_elems(91 + log_leaves, leaves * width).reshape(leaves, width)
    for k in {0, leaves // 3, leaves - 1}:
        cw[k, 0] = (2**48 - 0xdd5743e7f2a5a5d9) % GL_P
    d_cw, d_t = DeviceBuffer.from_numpy(gl, cw.reshape(-1)), DeviceBuffer(gl, 32 * (2 * leaves - 1))
    assert (gl.poseidon2_merkle_tree_ext2_ffi if ext else gl.poseidon2_merkle_tree_gl_ffi)(d_cw.ptr, d_t.ptr, leaves) == 0
    exp = np.zeros(4 * (2 * leaves - 1), dtype=np.uint64)
    oracle.oracle_bf_merkle_tree(cw.ctypes.data, leaves, int(ext), exp.ctypes.data)
    assert np.array_equal(d_t.to_numpy(), exp)


@pytest.mark.parametrize("log_leaves", [0, 1, 2, 3, 4, 6, 9, 13])
@pytest.mark.parametrize("ext", [False, True])
def test_small_monolith_trees(gl, oracle, log_leaves, ext):
    """Sixteen lanes a permutation and a warp a permutation, and (2^13 leaves) a layer a thread each in front of them; words at the ends of
    their range, and a leaf that needs the exact form: after the first linear layer (rows 4 and 5: 6 22 .., 7 6 ..) its words 4 and 5
    are 2^48 and 0, and 2^96 has no low word."""
    leaves, width = 1 << log_leaves, 4 if ext else 2
    cw = field_elems(191 + log_leaves, leaves * width).reshape(leaves, width)
    cw[0], cw[leaves // 2] = GL_P - 1, 2**32 - 1
    cw[leaves - 1] = 0
    y = pow(6 * 6 - 7 * 22, -1, GL_P) * -7 * 2**48 % GL_P   # 6 x + 22 y = 2^48, 7 x + 6 y = 0
    cw[leaves - 1, :2] = -6 * pow(7, -1, GL_P) * y % GL_P, y
    d_cw, d_t = DeviceBuffer.from_numpy(gl, cw.reshape(-1)), DeviceBuffer(gl, 32 * (2 * leaves - 1))
    assert (gl.monolith_merkle_tree_ext2_ffi if ext else gl.monolith_merkle_tree_gl_ffi)(d_cw.ptr, d_t.ptr, leaves) == 0
    exp = np.zeros(4 * (2 * leaves - 1), dtype=np.uint64)
    with pyoracle.merkle_hash(1):
        oracle.oracle_bf_merkle_tree(cw.ctypes.data, leaves, int(ext), exp.ctypes.data)
    assert np.array_equal(d_t.to_numpy(), exp)


@pytest.mark.parametrize("log_n,m", [(8, 6), (9, 6), (9, 9), (10, 8), (13, 12), (17, 17), (18, 6), (19, 12), (20, 15),
                                     (22, 6), (22, 7), (22, 9), (24, 10), (24, 11), (24, 13), (25, 11), (25, 12)])
def test_partial_evaluation_rows(oracle, gl, log_n, m):
    for lib, mod, fn, ofn in ((load_agl(), AGL_Q, load_agl().agl_partial_eval_ext2_from_base_ffi, oracle.oracle_agl_partial_eval_ext2_from_base),
                              (gl, GL_P, gl.partial_eval_ext2_from_gl_ffi, oracle.oracle_gl_partial_eval_ext2_from_base)):
        data, r = field_elems(40 + log_n, 1 << log_n, mod), field_elems(41 + m, 2 * m, mod)
        d_in, d_r, d_out = DeviceBuffer.from_numpy(lib, data), DeviceBuffer.from_numpy(lib, r), DeviceBuffer(lib, 8 << log_n)
        assert fn(d_in.ptr, d_out.ptr, d_r.ptr, log_n, m) == 0
        exp = np.zeros(2 << (log_n - m), dtype=np.uint64)
        ofn(data.ctypes.data, exp.ctypes.data, r.ctypes.data, log_n, m)
        assert np.array_equal(d_out.to_numpy()[:len(exp)], exp)


# rows of 2^10 elements, at most 2^12 of 2^8 or 2^9, or at most 2^11 shorter ones go by rows; many short rows took up to four times as
# long that way (2^24, m = 6)
@pytest.mark.parametrize("log_n,m,rows", [(8, 6, False), (9, 6, True), (17, 6, True), (18, 6, False), (18, 7, True), (19, 7, False),
                                          (20, 8, True), (21, 8, False), (21, 9, True), (22, 9, False), (22, 10, True)])
def test_partial_evaluation_route(oracle, gl, log_n, m, rows):
    for lib, mod, fn, ofn in ((load_agl(), AGL_Q, load_agl().agl_partial_eval_ext2_from_base_ffi, oracle.oracle_agl_partial_eval_ext2_from_base),
                              (gl, GL_P, gl.partial_eval_ext2_from_gl_ffi, oracle.oracle_gl_partial_eval_ext2_from_base)):
        data, r = field_elems(60 + log_n, 1 << log_n, mod), field_elems(61 + m, 2 * m, mod)
        d_in, d_r, d_out = DeviceBuffer.from_numpy(lib, data), DeviceBuffer.from_numpy(lib, r), DeviceBuffer(lib, 8 << log_n)
        buf = ctypes.create_string_buffer(4096)
        lib.mb_prof_enable(1)
        lib.mb_prof_reset()
        rc = fn(d_in.ptr, d_out.ptr, d_r.ptr, log_n, m)
        lib.mb_prof_report(buf, len(buf))
        lib.mb_prof_enable(0)
        assert rc == 0
        assert ("partial_eval_rows" in buf.value.decode()) == rows
        exp = np.zeros(2 << (log_n - m), dtype=np.uint64)
        ofn(data.ctypes.data, exp.ctypes.data, r.ctypes.data, log_n, m)
        assert np.array_equal(d_out.to_numpy()[:len(exp)], exp)


@pytest.mark.parametrize("n,planes", [(3, 2), (8, 1), (9, 4), (49 * 8, 3), (49 * 8 + 1, 2), (1999, 4), (25088, 1), (25089, 3)])
def test_tensor_core_commit_chunks(n, planes):
    """One wave of chunks, its last column, the first of the next; stages on both digit groups, odd counts of stages."""
    lib = load_agl()
    rng = np.random.default_rng(n + planes)
    dig = rng.integers(-127, 128, size=planes * n * 64, dtype=np.int8)
    dig[:64], dig[-64:] = 127, -127
    d_k, d_z, d_t = DeviceBuffer.from_numpy(lib, KEY), DeviceBuffer.from_numpy(lib, dig), DeviceBuffer(lib, lib.ajtai_tc_matrix_bytes(n))
    d_a, d_b, d_s = (DeviceBuffer(lib, planes * 42 * 64 * 8) for _ in range(3))
    assert lib.ajtai_materialize_tc_ffi(d_k.ptr, d_t.ptr, n, 0) == 0
    assert lib.ajtai_commit_s8_tiled_ffi(d_t.ptr, d_z.ptr, n, planes, d_a.ptr) == 0
    assert lib.ajtai_commit_s8_ffi(d_k.ptr, d_z.ptr, n, planes, 0, d_b.ptr) == 0
    if n < 500:
        want = pyoracle.ajtai_commit(KEY, dig, 1, n, planes)
    else:   # the scalar kernel, which has its own comparison with the oracle
        assert lib.ajtai_commit_s8_scalar_ffi(d_k.ptr, d_z.ptr, n, planes, 0, d_s.ptr) == 0
        want = d_s.to_numpy()
    assert np.array_equal(d_a.to_numpy(), want) and np.array_equal(d_b.to_numpy(), want)
    dig[(planes * n - 1) * 64 + 63] = -128   # the last digit of the last pair
    d_z = DeviceBuffer.from_numpy(lib, dig)
    assert lib.ajtai_commit_s8_tiled_ffi(d_t.ptr, d_z.ptr, n, planes, d_a.ptr) == -3
    assert lib.ajtai_commit_s8_ffi(d_k.ptr, d_z.ptr, n, planes, 0, d_b.ptr) == -3
