"""The word check for residue codes outside the alphabet (csrc/pb_codes.h),
built for the host, against the code-by-code rule: every byte value in every
position beside neighbours at the edges of the alphabet, and random words."""
import ctypes
import os
import random
import shutil
import subprocess

import pytest

HERE = os.path.dirname(__file__)
CSRC = os.path.join(HERE, "..", "parasail_b200", "csrc")
SOURCE = """
#include "pb_codes.h"
extern "C" uint32_t outside(uint32_t w, int L) { return codes_outside(w, L); }
"""


@pytest.fixture(scope="module")
def codes(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("codes")
    (d / "codes.cpp").write_text(SOURCE)
    so = str(d / "libcodes.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "codes.cpp")])
    lib = ctypes.CDLL(so)
    lib.outside.argtypes = [ctypes.c_uint32, ctypes.c_int]
    lib.outside.restype = ctypes.c_uint32
    return lib


@pytest.mark.parametrize("L", [1, 2, 4, 24, 32, 127, 128, 129, 200, 255, 256])
def test_word_check(codes, L):
    rng = random.Random(L)
    edge = [0, L - 1, min(L, 255), 127, 128, 255]
    words = [[c if k == at else rng.choice(edge) for k in range(4)] for at in range(4) for c in range(256)]
    words += [[c if k == at else 0 for k in range(4)] for at in range(4) for c in range(256)]
    words += [[rng.randrange(min(L, 256)) for _ in range(4)] for _ in range(500)]
    for b in words:
        w = sum(c << (8 * k) for k, c in enumerate(b))
        assert codes.outside(w, L) == sum(0x80 << (8 * k) for k, c in enumerate(b) if c >= L), b
