"""The batched sumcheck's state handle driven call by call: a fold without the round's message, claims asked for late,
alpha set again. Messages,
claims and finals against the oracle's proof, whose challenges the handle is given."""
import numpy as np
import pytest

from matrix_b200.ffi import DeviceBuffer, load_gl
from matrix_b200.sharded import GpuShard, e2_mul
from oracle import pyoracle

from .sharded_helpers import inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = load_gl()
    assert lib.goldilocks_cuda_init() == 0
    return lib


class Driven:
    """A handle on a whole (unsharded) instance set, and the oracle's proof of it."""

    def __init__(self, lib, K, nv):
        a, b, self.point = inputs(K, nv)
        self.K, self.nv = K, nv
        self.proof = pyoracle.batched_prove(a, b, np.array([c for t in self.point for c in t], dtype=np.uint64), K, nv)
        self.bufs = DeviceBuffer.from_numpy(lib, a), DeviceBuffer.from_numpy(lib, b)
        self.shard = GpuShard(lib, self.bufs[0].ptr, self.bufs[1].ptr, self.point, (1, 0), K, nv)
        self.alpha = tuple(int(x) for x in self.proof["alpha"])

    def check_message(self, rnd):
        assert np.array_equal(self.shard.round_message(), self.proof["round_msgs"][rnd].reshape(-1)), rnd

    def fold(self, rnd):
        self.shard.fold(tuple(int(x) for x in self.proof["challenges"][rnd]))

    def check_finals(self):
        want = self.proof["finals"].copy()
        pw = (1, 0)
        for k in range(self.K):   # the handle reports alpha^k a_k
            want[1 + k] = e2_mul(pw, tuple(int(x) for x in want[1 + k]))
            pw = e2_mul(pw, self.alpha)
        assert np.array_equal(self.shard.finals(), want.reshape(-1))
        self.shard.close()


# all rounds on the host from the start (K 2^n <= 1024), one pass, several passes with blocks of four, three and two rounds
@pytest.mark.parametrize("K,nv", [(1, 1), (1, 9), (1, 11), (1, 18), (3, 12), (16, 6), (16, 12)])
@pytest.mark.parametrize("asked", ["none", "last", "even", "odd", "thirds"])
def test_fold_without_message(lib, K, nv, asked):
    d = Driven(lib, K, nv)
    d.shard.set_alpha(d.alpha)
    for rnd in range(nv):
        if {"none": False, "last": rnd == nv - 1, "even": rnd % 2 == 0, "odd": rnd % 2 == 1, "thirds": rnd % 3 == 1}[asked]:
            d.check_message(rnd)
        d.fold(rnd)
    d.check_finals()


@pytest.mark.parametrize("K,nv", [(1, 1), (1, 9), (16, 12), (3, 17)])
@pytest.mark.parametrize("asked_at", ["after the first fold", "after the last fold", "before and after"])
def test_claims_after_a_fold(lib, K, nv, asked_at):
    d = Driven(lib, K, nv)
    want = d.proof["claims"].reshape(-1)
    if asked_at == "before and after":
        assert np.array_equal(d.shard.claims(), want)
    d.shard.set_alpha(d.alpha)
    for rnd in range(nv):
        d.fold(rnd)
        if rnd == 0 and asked_at != "after the last fold":
            assert np.array_equal(d.shard.claims(), want)
    assert np.array_equal(d.shard.claims(), want)
    d.check_finals()


@pytest.mark.parametrize("K,nv", [(2, 1), (1, 9), (16, 6), (16, 12), (3, 17)])
def test_alpha_set_again(lib, K, nv):
    """Before the first fold the last value counts, also when a message has been formed with another one; after it the call
    changes nothing."""
    d = Driven(lib, K, nv)
    d.shard.set_alpha((12345, 678))
    d.shard.round_message()
    d.shard.set_alpha(d.alpha)
    for rnd in range(nv):
        d.check_message(rnd)
        d.fold(rnd)
        d.shard.set_alpha((999 + rnd, 5))
    d.check_finals()
