"""The same-point prover at the sizes where its passes change: inside a word, one word, around the 256 words of a thread
block, uneven splits of the rounds, many leaves. Bit equality with the CPU prover."""
import numpy as np
import pytest

from oracle import pyoracle
from .test_same_point_gpu import gpu_prove, lib, random_instance   # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,arity,leaves", [(0, 2, 1), (0, 3, 2), (0, 5, 2), (0, 8, 3), (0, 10, 700), (0, 14, 2), (0, 15, 3),
                                               (0, 17, 2), (1, 5, 2), (1, 7, 300), (1, 15, 2), (1, 16, 1), (2, 4, 3), (2, 8, 2),
                                               (2, 9, 40), (2, 13, 1)])
def test_passes(lib, kind, arity, leaves):   # noqa: F811
    insts = [random_instance(40 + 11 * i, kind, arity) for i in range(leaves)]
    exp = pyoracle.agl_same_point_prove(insts, arity, b"sp-pass")
    got = gpu_prove(lib, insts, b"sp-pass")
    for key in ("round_msgs", "challenges", "f_evals", "final_eval", "state"):
        assert np.array_equal(got[key], exp[key]), key
