"""A pass that gave up a bounded wait, scratch that cannot be had, and the caller's way of waiting, seen from the host: the library's
own objects linked with a stand-in for the CUDA runtime, so no GPU is needed and none is made to fail."""
import ctypes
import os
import subprocess
import time

import numpy as np
import pytest

from matrix_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
MB_ERR_CUDA = -1
UNITS = ["gl_memory.cu", "prof.cu", "host/exchange.cu", "host/gl_batched_prover.cu", "agl_ajtai.cu"]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    objs = [os.path.join(build.OBJ, u.replace("/", "_") + ".o") for u in UNITS]
    fake = out[:-3] + ".o"
    subprocess.check_call(["gcc", "-O1", "-w", "-fPIC", "-c", os.path.join(HERE, "csrc", "fake_cudart.c"), "-o", fake])
    only = out[:-3] + ".map"   # statics of inline functions are unique in a process otherwise: the product's scratch pool would get these blocks
    with open(only, "w") as f:
        f.write("{ global: fake_*; gl_*; ajtai_*; local: *; };")
    subprocess.check_call(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-Wl,--version-script," + only, "-o", out] + objs + [fake, "-lrt", "-lpthread"])
    lib = ctypes.CDLL(out)
    u64 = ctypes.c_uint64
    lib.gl_batched_state_set_alpha.argtypes = lib.gl_batched_state_fold.argtypes = [ctypes.c_void_p, u64, u64]
    return lib


class Handle:
    """K instances of 2^nv words; the first pass runs on the tensor cores from K 2^nv = 2^14 on."""

    def __init__(self, lib, K, nv):
        self.lib, self.a, self.b = lib, np.ones(K << nv, dtype=np.uint64), np.ones(K << nv, dtype=np.uint64)
        self.pt, self.scale, self.out = np.ones(2 * nv, dtype=np.uint64), np.array([1, 0], dtype=np.uint64), np.zeros(2 * (2 * K + 1) + 8, dtype=np.uint64)
        self.h = ctypes.c_void_p()
        self.rc = lib.gl_batched_state_create(*(ctypes.c_void_p(x.ctypes.data) for x in (self.a, self.b, self.pt, self.scale)), K, nv,
                                              ctypes.byref(self.h))

    def claims(self):
        return self.lib.gl_batched_state_claims(self.h, ctypes.c_void_p(self.out.ctypes.data))

    def message(self):
        return self.lib.gl_batched_state_round_message(self.h, ctypes.c_void_p(self.out.ctypes.data))

    def fold(self):
        return self.lib.gl_batched_state_fold(self.h, 5, 7)

    def alpha(self):
        return self.lib.gl_batched_state_set_alpha(self.h, 3, 4)

    def finals(self):
        return self.lib.gl_batched_state_finals(self.h, ctypes.c_void_p(self.out.ctypes.data))

    def close(self):
        self.lib.gl_batched_state_destroy(self.h)


def test_first_pass(lib):
    lib.fake_fail_next_wait()
    s = Handle(lib, 1, 15)
    assert s.rc == 0 and s.alpha() == 0
    for _ in range(3):
        assert (s.claims(), s.message(), s.fold()) == (MB_ERR_CUDA,) * 3
    freed = lib.fake_scratch_freed()
    s.close()
    assert lib.fake_scratch_freed() == freed + 1   # its sums may not be zero: not for another proof


@pytest.mark.parametrize("K,nv,rounds", [(1, 16, 4), (1, 18, 7), (4, 14, 4), (16, 12, 3)])
def test_later_pass_and_every_call_after_it(lib, K, nv, rounds):
    """`rounds`: challenges after which the pass that fails is queued."""
    s = Handle(lib, K, nv)
    assert s.rc == 0 and s.alpha() == 0 and s.claims() == 0
    for r in range(rounds):
        if r == rounds - 1:
            lib.fake_fail_next_wait()
        assert s.message() == 0 and s.fold() == 0
    for r in range(rounds, nv + 2):   # on to the end and past it, whatever the caller makes of the errors
        assert s.message() != 0 and s.fold() != 0
    assert s.finals() != 0
    freed = lib.fake_scratch_freed()
    s.close()
    assert lib.fake_scratch_freed() == freed + 1


def test_scratch_is_kept_after_a_good_proof(lib):
    for _ in range(2):
        s = Handle(lib, 2, 13)
        assert s.rc == 0 and s.alpha() == 0 and s.claims() == 0
        for _ in range(13):
            assert s.message() == 0 and s.fold() == 0
        assert s.finals() == 0
        counts = lib.fake_scratch_allocated(), lib.fake_scratch_freed()
        s.close()
        assert (lib.fake_scratch_allocated(), lib.fake_scratch_freed()) == counts
    s = Handle(lib, 2, 13)
    assert lib.fake_scratch_allocated() == counts[0]
    s.close()


@pytest.mark.parametrize("planes", [1, 3, 4, 5, 9])   # one pass over the matrix, and several
def test_ajtai_commitment_without_scratch(lib, planes):
    """A commitment needs a scratch block for nothing but an earlier answer: without one it synchronises."""
    allocated, holders = lib.fake_scratch_allocated(), []
    while lib.fake_scratch_allocated() == allocated:   # every block kept from earlier proofs is in use
        holders.append(Handle(lib, 1, 12))
    key, digits, out = np.ones(8, dtype=np.uint32), np.ones(40 * 64 * planes, dtype=np.int8), np.zeros(42 * 64 * planes, dtype=np.uint64)
    args = [ctypes.c_void_p(x.ctypes.data) for x in (key, digits)] + [ctypes.c_uint64(40), planes, ctypes.c_uint64(0), ctypes.c_void_p(out.ctypes.data)]
    before = lib.fake_synchronised()
    lib.fake_no_scratch(1)
    rcs = [lib.ajtai_commit_s8_ffi(*args) for _ in range(2)]
    lib.fake_no_scratch(0)
    assert rcs == [0, 0] and lib.fake_synchronised() == before + 2
    for h in holders:
        h.close()
    assert lib.ajtai_commit_s8_ffi(*args) == 0


def test_waits_of_a_caller_that_does_not_spin(lib):
    """Device flags of blocking synchronisation (4) or yielding (2): a wait for words is the synchronisation that they are for. No word
    arrives here, so the others (0 and 1) use up their polls, a third of a millisecond or more each, in front of it."""
    key, digits, out = np.ones(8, dtype=np.uint32), np.ones(8 * 64, dtype=np.int8), np.zeros(42 * 64, dtype=np.uint64)
    args = [ctypes.c_void_p(x.ctypes.data) for x in (key, digits)] + [ctypes.c_uint64(8), 1, ctypes.c_uint64(0), ctypes.c_void_p(out.ctypes.data)]
    took = {}
    for flags in (0, 1, 2, 4, 4 | 8):   # 8: mapped host memory, no way of waiting
        lib.fake_device_flags(flags)
        assert lib.ajtai_commit_s8_ffi(*args) == 0
        before, t = lib.fake_synchronised(), time.thread_time()
        for _ in range(40):
            assert lib.ajtai_commit_s8_ffi(*args) == 0
        took[flags] = time.thread_time() - t
        assert lib.fake_synchronised() == before + 40
    lib.fake_device_flags(0)
    assert max(took[2], took[4], took[12]) < min(took[0], took[1]) / 4, took
