"""Reductions without their rare repairs: every one that is left out is told of, and few others are, because a permutation that is
told of one runs again."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

from matrix_b200 import build, load_gl
from matrix_b200.ffi import DeviceBuffer

from .conftest import GL_P, field_elems

HERE = os.path.dirname(os.path.abspath(__file__))
SRC, OUT = os.path.join(HERE, "csrc", "missed_check.cu"), os.path.join(HERE, "csrc", "_build", "libmissed_check.so")


def _library():
    deps = [SRC] + [os.path.join(dp, f) for dp, _, fs in os.walk(build.CSRC) for f in fs if f.endswith((".cuh", ".hpp"))]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.check_call([build.NVCC] + build.ARCH + build.FLAGS + ["-I", build.CSRC, "-shared", "-o", OUT, SRC])
    return ctypes.CDLL(OUT)


def test_builds():
    _library()


@pytest.fixture(scope="module")
def lib():
    return _library()


@pytest.fixture(scope="module")
def gl():
    lib = load_gl()
    assert lib.goldilocks_cuda_init() == 0
    return lib


def _run(gl, call, rows):
    d_in = DeviceBuffer.from_numpy(gl, np.array(rows, dtype=np.uint32).reshape(-1).view(np.uint64))
    d_out = DeviceBuffer(gl, 16 * len(rows))
    assert call(ctypes.c_void_p(d_in.ptr), ctypes.c_void_p(d_out.ptr), len(rows)) == 0
    return d_out.to_numpy().reshape(-1, 2)


def _look(values, out, most_told):
    told = 0
    for v, (word, missed) in zip(values, out):
        told += int(missed)
        assert missed or int(word) % GL_P == v % GL_P, hex(v)
    assert told <= most_told


EDGE = [0, 1, 2, 31, 32, 2**31, 2**32 - 33, 2**32 - 32, 2**32 - 2, 2**32 - 1]


@pytest.mark.gpu
@pytest.mark.parametrize("most", [0, 1, 3, 29, 31])
def test_reductions(gl, lib, most):
    rng = np.random.default_rng(5 + most)
    rows = [z + (z4, most) for z in itertools.product(EDGE, repeat=4) for z4 in {0, most // 2, most}]
    edges = len(rows)
    rows += [tuple(int(x) for x in rng.integers(0, 2**32, 4)) + (int(rng.integers(0, most + 1)), most) for _ in range(40000)]
    _look([sum(z << (32 * i) for i, z in enumerate(r[:5])) for r in rows], _run(gl, lib.mc_reduce, rows), edges)   # none of the random ones


@pytest.mark.gpu
def test_sums(gl, lib):
    rng = np.random.default_rng(6)
    rows = [(a, b, c) for a, b in itertools.product(EDGE, repeat=2) for c in (0, 1, 2, 7, 160, 1023)]
    edges = len(rows)
    rows += [tuple(int(x) for x in rng.integers(0, 2**32, 2)) + (int(rng.integers(0, 1024)),) for _ in range(40000)]
    _look([a + (b << 32) + (c << 64) for a, b, c in rows], _run(gl, lib.mc_sum, rows), edges)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [8, 12])
def test_permutations_that_run_again(gl, lib, width):
    """2^22 permutations of at most 700 reductions each, of which one in 2^32 looks like a repair and fewer need one: one or two in
    all. A bound of six (a Poisson count of 1.4 is above it once in a thousand, and the states are always the same)."""
    n = 1 << 22
    d_in, d_count = DeviceBuffer.from_numpy(gl, field_elems(300 + width, width * n)), DeviceBuffer.from_numpy(gl, np.zeros(1, dtype=np.uint64))
    assert lib.mc_permute(width, ctypes.c_void_p(d_in.ptr), n, ctypes.c_void_p(d_count.ptr)) == 0
    again, wrong = d_count.to_numpy().view(np.uint32)
    assert wrong == 0 and again <= 6
