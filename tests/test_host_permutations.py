"""Both forms of every host permutation (portable, and the one for this core's instruction set) against the oracle."""
import ctypes
import random

import pytest

from matrix_b200.inputs import AGL_Q
from .conftest import GL_P

RC0 = 0xdd5743e7f2a5a5d9   # Poseidon2's first constant of lane 0


def test_device_tables_are_aligned(hostcheck):
    """The tables of the tiles and of the permutation a warp are copied by 16-byte loads: their type has to say so, or where they lie
    depends on their neighbours in the translation unit."""
    o = (ctypes.c_size_t * 4)()
    hostcheck.hc_p2_tables(o)
    assert o[0] >= 16 and o[2] >= 16 and o[1] % 16 == 0 and o[3] % 16 == 0


def _states(width, p):
    rnd = random.Random(31)
    edge = [0, 1, p - 1, p, 2**64 - 1, 2**32 - 1, 2**32, 2**63]
    yield from ([e] * width for e in edge)
    # squares with a low word below the top limb: the first S-box sees 2^48 (2^96 has no low word) and neighbours
    yield from ([(v - RC0) % GL_P] * width for v in (2**48, 2**48 + 1, 2**63, 2**33 * 3))
    for _ in range(60):
        yield [rnd.choice(edge) if rnd.random() < 0.3 else rnd.randrange(2**64) for _ in range(width)]


@pytest.mark.parametrize("name,width,p,want", [
    ("hc_poseidon2_host", 8, GL_P, "gl_poseidon2_permute"),
    ("hc_gl_monolith_host", 12, GL_P, "oracle_gl_monolith_permute"),
    ("hc_agl_monolith", 12, AGL_Q, "oracle_agl_monolith_permute")])
def test_host_permutation_forms(hostcheck, oracle, name, width, p, want):
    words = ctypes.c_uint64 * width
    for state in _states(width, p):
        expect = words(*[w % p for w in state])
        getattr(oracle, want)(expect)
        for form in (name, name + "_portable"):
            got = words(*state)
            getattr(hostcheck, form)(got)
            assert list(got) == list(expect), (form, state)
