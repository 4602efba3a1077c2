"""What the tensor-core kernels do once a bounded wait has run out: units of the library built with no polls at all, so that every
wait inside a kernel runs out at once (none is left waiting, and what was issued is still drained). Rows of a partial
evaluation and hashes are formed again from memory; a proof fails, on every call, and the next one is right."""
import ctypes
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from matrix_b200 import build, ffi
from matrix_b200.ffi import DeviceBuffer

from .conftest import field_elems

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.join(HERE, "csrc", "_build", "libexpired_waits.so")
UNITS = ["gl_memory.cu", "prof.cu", "gl_merkle.cu", "gl_basefold.cu", "host/exchange.cu", "host/gl_sumcheck_prover.cu",
         "host/gl_batched_prover.cu"]
MB_ERR_CUDA = -1


def _library():
    deps = [os.path.join(dp, f) for dp, _, fs in os.walk(build.CSRC) for f in fs]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        objs = [os.path.join(os.path.dirname(OUT), "expired_" + u.replace("/", "_") + ".o") for u in UNITS]
        cc = [build.NVCC] + build.ARCH + build.FLAGS + ["-DMB_TC_POLLS=0", "-I", build.CSRC, "-c"]
        with ThreadPoolExecutor(len(UNITS)) as ex:
            list(ex.map(lambda uo: subprocess.check_call(cc + [os.path.join(build.CSRC, uo[0]), "-o", uo[1]]), zip(UNITS, objs)))
        subprocess.check_call([build.NVCC] + build.ARCH + ["-shared", "-ccbin", "g++", "-o", OUT] + objs)
        for o in objs:
            os.remove(o)
    lib = ctypes.CDLL(OUT)
    for name, (res, args) in ffi.gl_signatures().items():
        fn = getattr(lib, name, None)
        if fn is not None:
            fn.restype, fn.argtypes = res, args
    return lib


def test_units_build():
    _library()


@pytest.fixture(scope="module")
def lib():
    lib = _library()
    assert lib.goldilocks_cuda_init() == 0
    return lib


# clusters of one, two and four blocks; more than one tile a block
@pytest.mark.gpu
@pytest.mark.parametrize("log_n,m", [(22, 7), (24, 11), (24, 12)])
def test_rows_are_formed_again(lib, oracle, log_n, m):
    data, r = field_elems(140 + log_n, 1 << log_n), field_elems(141 + m, 2 * m)
    d_in, d_r, d_out = DeviceBuffer.from_numpy(lib, data), DeviceBuffer.from_numpy(lib, r), DeviceBuffer(lib, 8 << log_n)
    assert lib.partial_eval_ext2_from_gl_ffi(d_in.ptr, d_out.ptr, d_r.ptr, log_n, m) == 0
    exp = np.zeros(2 << (log_n - m), dtype=np.uint64)
    oracle.oracle_gl_partial_eval_ext2_from_base(data.ctypes.data, exp.ctypes.data, r.ctypes.data, log_n, m)
    assert np.array_equal(d_out.to_numpy()[:len(exp)], exp)


@pytest.mark.gpu
@pytest.mark.parametrize("ext", [False, True])
def test_hashes_are_formed_again(lib, oracle, ext):
    leaves, width = 1 << 20, 4 if ext else 2
    cw = field_elems(178, leaves * width)
    d_cw, d_t = DeviceBuffer.from_numpy(lib, cw), DeviceBuffer(lib, 32 * (2 * leaves - 1))
    assert (lib.poseidon2_merkle_tree_ext2_ffi if ext else lib.poseidon2_merkle_tree_gl_ffi)(d_cw.ptr, d_t.ptr, leaves) == 0
    exp = np.zeros(4 * (2 * leaves - 1), dtype=np.uint64)
    oracle.oracle_bf_merkle_tree(cw.ctypes.data, leaves, int(ext), exp.ctypes.data)
    assert np.array_equal(d_t.to_numpy(), exp)


def _prove(lib, d, nv, base, polys):
    out = [np.zeros(n, dtype=np.uint64) for n in (nv * (d + 1) * 2, 2 * nv, 2 * d, 2)]
    buf = DeviceBuffer.from_numpy(lib, polys)
    rc = lib.gl_sumcheck_prove_device_ffi(buf.ptr, d, nv, base, b"waits", 5, *(o.ctypes.data for o in out), None)
    return rc, out


# base and extension tables, with and without a fold in the pass that fails (the first one does)
@pytest.mark.gpu
@pytest.mark.parametrize("d,nv,base,small", [(2, 15, 1, 13), (2, 15, 0, 13), (3, 16, 1, 13), (3, 16, 0, 13)])
def test_a_proof_fails_and_the_next_is_right(lib, oracle, d, nv, base, small):
    from oracle import pyoracle
    words = 1 if base else 2
    assert _prove(lib, d, nv, base, field_elems(150 + d, (d << nv) * words))[0] == MB_ERR_CUDA
    polys = field_elems(151 + d, (d << small) * words)   # no pass on the tensor cores, but sums over blocks
    rc, out = _prove(lib, d, small, base, polys)
    exp = pyoracle.sumcheck_prove(polys, d, small, bool(base), b"waits")
    assert rc == 0 and np.array_equal(out[0], exp["round_msgs"].reshape(-1)) and np.array_equal(out[3], exp["final_eval"].reshape(-1))


# the first pass (weights) of one instance and of sixteen; the first is right and the second, which folds, fails; every later call
# fails too
@pytest.mark.gpu
@pytest.mark.parametrize("K,nv,good", [(1, 15, 0), (16, 12, 0), (64, 10, 2)])
def test_a_state_stays_failed(lib, K, nv, good):
    a, b = (DeviceBuffer.from_numpy(lib, field_elems(160 + i, K << nv)) for i in range(2))
    pt, scale, out, h = field_elems(162, 2 * nv), np.array([1, 0], dtype=np.uint64), np.zeros(4 * K + 8, dtype=np.uint64), ctypes.c_void_p()
    assert lib.gl_batched_state_create(a.ptr, b.ptr, pt.ctypes.data, scale.ctypes.data, K, nv, ctypes.byref(h)) == 0
    assert lib.gl_batched_state_set_alpha(h, 3, 4) == 0
    for _ in range(good):
        assert lib.gl_batched_state_claims(h, out.ctypes.data) == 0
        assert lib.gl_batched_state_round_message(h, out.ctypes.data) == 0
        assert lib.gl_batched_state_fold(h, 5, 7) == 0
    for _ in range(2):
        assert lib.gl_batched_state_claims(h, out.ctypes.data) == (0 if good else MB_ERR_CUDA)   # kept since the first pass
        assert lib.gl_batched_state_round_message(h, out.ctypes.data) == MB_ERR_CUDA
        assert lib.gl_batched_state_fold(h, 5, 7) == MB_ERR_CUDA
    lib.gl_batched_state_destroy(h)
