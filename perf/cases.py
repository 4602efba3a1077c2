"""What the prover path is timed on: whole calls of the public entry points, over the sizes they are used at.

Operations (a case's "op"):

  sumcheck    one proof of sum_x prod_i f_i(x), the tables resident on the device
              (gl_sumcheck_prove_device_ffi, agl_sumcheck_prove_device_ffi)
  verify      the host verifier of such a proof (gl_sumcheck_verify_ffi)
  basefold    commitment and opening of one multilinear polynomial, evaluations on the device
              (basefold_commit_device + basefold_open_ext2) or in page-locked host memory (basefold_prove_host)
  ajtai       ring commitment of signed 8-bit digit planes, the matrix regenerated from the ChaCha8 stream
              (ajtai_commit_s8_ffi) or laid out once in operand order (ajtai_commit_s8_tiled_ffi)
  batched     K instances of eq * a * b under one challenge (gl_batched_prove_sharded with one rank)
  same_point  the fold tree's same-point sumcheck over packed binary or ternary witnesses
              (agl_same_point_prove_device_ffi)
  einsum      one einsum block of a decoder layer: operand partial evaluations, eq table, sumcheck
              (agl_einsum_prove_device_ffi)

Every result is a vector of field elements or bytes and has exactly one right value.
"""
import ctypes
import math

import numpy as np
import torch

from matrix_b200 import load_gl
from matrix_b200.ffi import load_agl
from matrix_b200.inputs import AGL_Q, GL_P, field_elems
from matrix_b200.layer_trace import EinsumPlan, LayerProver, prove_einsum_native
from matrix_b200.sharded import prove_batched_native

LABEL = b"perf-cases"
AJTAI_ROWS = 42 * 64      # output coefficients of one plane
DEGREE = 64               # coefficients of a ring element
HASH_MULTS = {"poseidon2": 520, "monolith": 120}   # field multiplications of one permutation, about


def listed():
    return [
        # a lookup or bias table: ten rounds whose tables fit one SM, so launches and the transcript are the proof
        dict(name="sumcheck_1k", op="sumcheck", field="gl", num_vars=10, degree=2, base=True),
        # f * g over 2^20 uniform field elements each: the single sumcheck the benchmark names
        dict(name="sumcheck_1m", op="sumcheck", field="gl", num_vars=20, degree=2, base=True),
        # eq * a * b on extension tables of 2^22 points: a gate of the other field, after a first folding layer
        dict(name="sumcheck_4m_ext_cubic", op="sumcheck", field="agl", num_vars=22, degree=3, base=False),
        # the other side of the protocol: a verifier replays the 2^20 proof on a host core
        dict(name="verify_1m", op="verify", num_vars=20, degree=2),
        # a small polynomial (a norm's weights): every tree is latency bound
        dict(name="basefold_4k", op="basefold", num_vars=12, log_rate=1, hash="poseidon2", queries=100, source="device"),
        # a vocabulary shard with the other tree hash, rate 1/4, from host memory
        dict(name="basefold_1m_monolith_host", op="basefold", num_vars=20, log_rate=2, hash="monolith", queries=64, source="host"),
        # the headline: 2^24 evaluations, rate 1/2, 100 queries
        dict(name="basefold_16m", op="basefold", num_vars=24, log_rate=1, hash="poseidon2", queries=100, source="device"),
        # one activation tensor (97 tokens of 4096 values, rows padded to ring elements) against a resident matrix
        dict(name="ajtai_activation", op="ajtai", columns=6209, planes=3, matrix="tiled"),
        # a weight tensor of 2^24 coefficients, the matrix from its seed
        dict(name="ajtai_weight", op="ajtai", columns=1 << 18, planes=3, matrix="seed"),
        # sixteen gates under one random combination
        dict(name="batched_16x4m", op="batched", num_vars=22, instances=16),
        # one node of the fold tree: 42 packed binary leaves of arity 22
        dict(name="same_point_42x4m", op="same_point", arity=22, leaves=42, witness="binary"),
        # an attention projection of a decoder layer: 128 tokens, 4096 x 4096 weights
        dict(name="einsum_projection", op="einsum", equation="si,ij->sj", s=7, i=12, j=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["sumcheck", "sumcheck", "verify", "basefold", "basefold", "ajtai", "ajtai", "batched", "same_point",
                     "einsum", "einsum"])
    if op == "sumcheck":
        base, degree = rng.random() < 0.5, rng.randint(1, 4)
        top = 24 if base and degree <= 2 else 22
        return dict(op=op, field=rng.choice(["gl", "agl"]), num_vars=rng.randint(6, top), degree=degree, base=base)
    if op == "verify":
        return dict(op=op, num_vars=rng.randint(6, 22), degree=rng.randint(1, 4))
    if op == "basefold":
        log_rate = rng.randint(1, 3)
        return dict(op=op, num_vars=rng.randint(8, 24 - log_rate), log_rate=log_rate, hash=rng.choice(["poseidon2", "monolith"]),
                    queries=rng.randint(16, 128), source=rng.choice(["device", "host"]))
    if op == "ajtai":
        return dict(op=op, columns=_log_int(rng, 64, 1 << 18) | 1, planes=rng.randint(1, 4), matrix=rng.choice(["tiled", "seed"]))
    if op == "batched":
        return dict(op=op, num_vars=rng.randint(10, 21), instances=rng.randint(2, 24))
    if op == "same_point":
        return dict(op=op, arity=rng.randint(8, 21), leaves=rng.randint(2, 56), witness=rng.choice(["binary", "ternary"]))
    eq = rng.choice(["si,ij->sj", "hsd,htd->hst", "hst,htd->hsd", "si,si->si"])
    if eq == "si,ij->sj":
        return dict(op=op, equation=eq, s=rng.randint(3, 9), i=rng.randint(6, 12), j=rng.randint(6, 12))
    if eq == "si,si->si":
        return dict(op=op, equation=eq, s=rng.randint(3, 9), i=rng.randint(6, 12))
    return dict(op=op, equation=eq, h=rng.randint(2, 5), s=rng.randint(4, 8), t=rng.randint(4, 8), d=rng.randint(5, 7))


class State:
    """The buffers and handles a caller keeps for one case; handles go back to the library with the object."""

    def __init__(self, case, lib):
        self.case, self.lib, self._destroy = case, lib, []

    def own(self, destroy, handle):
        self._destroy.append((destroy, handle))
        return handle

    def __del__(self):
        for destroy, handle in self._destroy:
            destroy(handle)


def _check(rc, what):
    if rc != 0:
        raise RuntimeError("%s returned %d" % (what, rc))


def _words(n):
    return np.zeros(n, dtype=np.uint64)


def _uniform(lib, n, seed, modulus):
    """n uniform residues below `modulus` on the device, one 64-bit word each."""
    t = torch.empty(n, dtype=torch.int64, device="cuda")
    _check(lib.mb_fill_splitmix(t.data_ptr(), n, seed * 0x9E3779B97F4A7C15 % (1 << 64), modulus), "mb_fill_splitmix")
    return t


def _einsum_dims(case):
    return {c: case[c] for c in "siijhtd" if c in case}


# ---- preparation -------------------------------------------------------------------------------

def _prepare_sumcheck(case, seed):
    lib = load_gl() if case["field"] == "gl" else load_agl()
    s = State(case, lib)
    nv, d = case["num_vars"], case["degree"]
    s.tables = _uniform(lib, (d << nv) * (1 if case["base"] else 2), seed, GL_P if case["field"] == "gl" else AGL_Q)
    s.msgs, s.challenges, s.finals, s.final = _words(nv * (d + 1) * 2), _words(nv * 2), _words(2 * d), _words(2)
    return s


def _run_sumcheck(s):
    nv, d, base = s.case["num_vars"], s.case["degree"], int(s.case["base"])
    out = (s.msgs.ctypes.data, s.challenges.ctypes.data, s.finals.ctypes.data, s.final.ctypes.data)
    if s.case["field"] == "gl":
        rc = s.lib.gl_sumcheck_prove_device_ffi(s.tables.data_ptr(), d, nv, base, LABEL, len(LABEL), *out, None)
    else:
        t = ctypes.c_void_p()
        _check(s.lib.agl_transcript_create(LABEL, len(LABEL), ctypes.byref(t)), "agl_transcript_create")
        rc = s.lib.agl_sumcheck_prove_device_ffi(s.tables.data_ptr(), d, nv, base, t, *out)
        s.lib.agl_transcript_destroy(t)
    _check(rc, "sumcheck")
    return [s.msgs, s.challenges, s.finals, s.final]


def _prepare_verify(case, seed):
    s = _prepare_sumcheck(dict(case, field="gl", base=True), seed)
    _run_sumcheck(s)
    s.tables = None   # a verifier has the proof only
    first = [int(w) for w in s.msgs[:4]]
    s.claim = np.array([(first[0] + first[2]) % GL_P, (first[1] + first[3]) % GL_P], dtype=np.uint64)
    s.replayed, s.ok = _words(2 * case["num_vars"]), ctypes.c_int()
    return s


def _run_verify(s):
    _check(s.lib.gl_sumcheck_verify_ffi(s.msgs.ctypes.data, s.final.ctypes.data, s.claim.ctypes.data, s.case["degree"],
                                        s.case["num_vars"], LABEL, len(LABEL), s.replayed.ctypes.data, ctypes.byref(s.ok)), "verify")
    return [s.replayed, s.ok.value]


def _prepare_basefold(case, seed):
    lib = load_gl()
    s = State(case, lib)
    nv, lr = case["num_vars"], case["log_rate"]
    s.evals = _uniform(lib, 1 << nv, seed, GL_P)
    if case["source"] == "host":
        host = torch.empty(1 << nv, dtype=torch.int64, pin_memory=True)
        host.copy_(s.evals)
        s.evals = host
    s.point = field_elems(seed, 2 * nv)
    s.table = ctypes.c_void_p()
    _check(lib.basefold_table_create(nv, lr, nv, 42, ctypes.byref(s.table)), "basefold_table_create")
    s.own(lib.basefold_table_destroy, s.table)
    s.root = _words(4)
    s.proof = torch.zeros(lib.basefold_proof_words(nv, lr, case["queries"]), dtype=torch.int64, pin_memory=True)
    return s


def _run_basefold(s):
    c, lib = s.case, s.lib
    nv, lr, nq = c["num_vars"], c["log_rate"], c["queries"]
    _check(lib.basefold_set_merkle_hash(1 if c["hash"] == "monolith" else 0), "basefold_set_merkle_hash")
    if c["source"] == "host":
        _check(lib.basefold_prove_host(s.evals.data_ptr(), nv, lr, s.point.ctypes.data, s.table, LABEL, len(LABEL), nq,
                                       s.root.ctypes.data, s.proof.data_ptr()), "basefold_prove_host")
    else:
        h = ctypes.c_void_p()
        _check(lib.basefold_commit_device(s.evals.data_ptr(), nv, lr, ctypes.byref(h), s.root.ctypes.data), "basefold_commit_device")
        rc = lib.basefold_open_ext2(h, s.point.ctypes.data, s.table, LABEL, len(LABEL), nq, s.proof.data_ptr(), None)
        lib.basefold_commitment_destroy(h)
        _check(rc, "basefold_open_ext2")
    return [s.root, s.proof]


def _prepare_ajtai(case, seed):
    lib = load_agl()
    s = State(case, lib)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, planes = case["columns"], case["planes"]
    s.digits = torch.randint(-127, 128, (planes * n * DEGREE,), dtype=torch.int8, device="cuda", generator=gen)
    s.key = torch.arange(1, 9, dtype=torch.int32, device="cuda")   # the commitment key is public and fixed
    s.matrix = None
    if case["matrix"] == "tiled":
        s.matrix = torch.empty(lib.ajtai_tc_matrix_bytes(n), dtype=torch.uint8, device="cuda")
        torch.cuda.current_stream().synchronize()
        _check(lib.ajtai_materialize_tc_ffi(s.key.data_ptr(), s.matrix.data_ptr(), n, 0), "ajtai_materialize_tc_ffi")
    s.out = torch.zeros(planes * AJTAI_ROWS, dtype=torch.int64, device="cuda")
    return s


def _run_ajtai(s):
    n, planes = s.case["columns"], s.case["planes"]
    if s.matrix is not None:
        rc = s.lib.ajtai_commit_s8_tiled_ffi(s.matrix.data_ptr(), s.digits.data_ptr(), n, planes, s.out.data_ptr())
    else:
        rc = s.lib.ajtai_commit_s8_ffi(s.key.data_ptr(), s.digits.data_ptr(), n, planes, 0, s.out.data_ptr())
    _check(rc, "ajtai commit")
    return [s.out]


def _prepare_batched(case, seed):
    lib = load_gl()
    s = State(case, lib)
    n = case["instances"] << case["num_vars"]
    s.a, s.b = _uniform(lib, n, 2 * seed, GL_P), _uniform(lib, n, 2 * seed + 1, GL_P)
    pt = field_elems(seed, 2 * case["num_vars"])
    s.point = [(int(pt[2 * i]), int(pt[2 * i + 1])) for i in range(case["num_vars"])]
    exchange = (ctypes.c_void_p * 1)()
    _check(lib.mb_exchange_local_create(1, exchange), "mb_exchange_local_create")
    s.exchange = s.own(lib.mb_exchange_destroy, exchange[0])
    return s


def _run_batched(s):
    return prove_batched_native(s.lib, s.exchange, s.a.data_ptr(), s.b.data_ptr(), s.case["instances"], s.case["num_vars"],
                                s.point, LABEL)


def _prepare_same_point(case, seed):
    lib = load_agl()
    s = State(case, lib)
    arity, leaves = case["arity"], case["leaves"]
    words = max(1, (1 << arity) >> 6)
    s.kind = 1 if case["witness"] == "ternary" else 0
    s.w0 = _uniform(lib, leaves * words, 2 * seed, 0xFFFFFFFFFFFFFFFF)
    s.w1 = None
    if s.kind:   # masks of the +1 and the -1 coefficients
        s.w1 = _uniform(lib, leaves * words, 2 * seed + 1, 0xFFFFFFFFFFFFFFFF)
        s.w1 &= ~s.w0
    torch.cuda.current_stream().synchronize()
    s.points = field_elems(seed, 2 * arity * leaves, AGL_Q)
    s.values = _words(2 * leaves)
    _check(lib.agl_same_point_claims_device_ffi(leaves, arity, s.points.ctypes.data, s.kind, s.w0.data_ptr(),
                                                s.w1.data_ptr() if s.kind else None, s.values.ctypes.data), "claims")
    s.msgs, s.challenges, s.reveals, s.final = _words(6 * arity), _words(2 * arity), _words(2 * leaves), _words(2)
    return s


def _run_same_point(s):
    t = ctypes.c_void_p()
    _check(s.lib.agl_transcript_create(LABEL, len(LABEL), ctypes.byref(t)), "agl_transcript_create")
    rc = s.lib.agl_same_point_prove_device_ffi(s.case["leaves"], s.case["arity"], s.points.ctypes.data, s.values.ctypes.data,
                                               s.kind, s.w0.data_ptr(), s.w1.data_ptr() if s.kind else None, t,
                                               s.msgs.ctypes.data, s.challenges.ctypes.data, s.reveals.ctypes.data,
                                               s.final.ctypes.data)
    s.lib.agl_transcript_destroy(t)
    _check(rc, "agl_same_point_prove_device_ffi")
    return [s.msgs, s.challenges, s.reveals, s.final]


def _prepare_einsum(case, seed):
    lib = load_agl()
    s = State(case, lib)
    s.prover, s.dims = LayerProver(lib), _einsum_dims(case)
    pl = EinsumPlan(case["equation"], s.dims)
    # 16-bit fixed point values as field elements: what quantised weights and activations are
    s.operands = [_uniform(lib, 1 << sum(s.dims[c] for c in t), 8 * seed + j, 1 << 16) for j, t in enumerate(pl.inputs)]
    n_out = sum(s.dims[c] for c in pl.out)
    s.point = field_elems(seed, 2 * n_out, AGL_Q).reshape(n_out, 2)
    s.prover.plan(case["equation"], s.dims)   # index tables: once per equation and shape
    return s


def _run_einsum(s):
    t = ctypes.c_void_p()
    _check(s.lib.agl_transcript_create(LABEL, len(LABEL), ctypes.byref(t)), "agl_transcript_create")
    out = prove_einsum_native(s.prover, s.case["equation"], s.dims, [o.data_ptr() for o in s.operands], s.point, t)
    s.lib.agl_transcript_destroy(t)
    return list(out)


_PREPARE = dict(sumcheck=_prepare_sumcheck, verify=_prepare_verify, basefold=_prepare_basefold, ajtai=_prepare_ajtai,
                batched=_prepare_batched, same_point=_prepare_same_point, einsum=_prepare_einsum)
_RUN = dict(sumcheck=_run_sumcheck, verify=_run_verify, basefold=_run_basefold, ajtai=_run_ajtai, batched=_run_batched,
            same_point=_run_same_point, einsum=_run_einsum)


def prepare(case, seed):
    return _PREPARE[case["op"]](case, seed)


def run(state):
    return _RUN[state.case["op"]](state)


# ---- work and tolerance --------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once. "flops": 64-bit modular multiplications of the protocol's textbook
    form (one each), and for the Ajtai commitment 8-bit multiply-adds (two each)."""
    op = case["op"]
    if op in ("sumcheck", "verify"):
        nv, d = case["num_vars"], case["degree"]
        proof = 16 * (nv * (d + 2) + d + 1)
        if op == "verify":
            return {"bytes": 2 * proof, "flops": HASH_MULTS["poseidon2"] * 8.0 * nv * (d + 2)}
        return {"bytes": (d << nv) * (8 if case["base"] else 16) + proof, "flops": 4.0 * (d + (d + 1) * max(d - 1, 1)) * (1 << nv)}
    if op == "basefold":
        nv, lr, nq = case["num_vars"], case["log_rate"], case["queries"]
        code = 1 << (nv + lr)
        proof = 8 * load_gl().basefold_proof_words(nv, lr, nq)
        permutations = (1 << nv) + code   # the commitment's tree over one block of the repetition code, the folded trees
        # the evaluations and the folding table are read, the codeword kept for later openings
        return {"bytes": (8 << nv) + 16 * code + 8 * code + proof,
                "flops": float(HASH_MULTS[case["hash"]] * permutations + 8 * code)}
    if op == "ajtai":
        n, planes = case["columns"], case["planes"]
        matrix = 42 * DEGREE * 8 * n if case["matrix"] == "tiled" else 32
        return {"bytes": n * DEGREE * planes + matrix + 8 * planes * AJTAI_ROWS, "flops": 2.0 * AJTAI_ROWS * DEGREE * 8 * n * planes}
    if op == "batched":
        k, nv = case["instances"], case["num_vars"]
        return {"bytes": (16 * k << nv) + 16 * (5 * nv + 3 * k), "flops": 24.0 * k * (1 << nv)}
    if op == "same_point":
        m, arity = case["leaves"], case["arity"]
        masks = 2 if case["witness"] == "ternary" else 1
        return {"bytes": masks * m * max(8, (1 << arity) >> 3) + 16 * m * (arity + 2) + 64 * arity, "flops": 12.0 * m * (1 << arity)}
    dims = _einsum_dims(case)
    pl = EinsumPlan(case["equation"], dims)
    read = sum(1 << sum(dims[c] for c in t) for t in pl.inputs)
    d = len(pl.inputs) + 1
    return {"bytes": 8 * read + 16 * pl.rounds * (d + 2), "flops": 2.0 * read + 4.0 * (d * d + d) * (1 << pl.rounds)}


def tolerance(case):
    return "exact"
