"""The split of a batch's CIGARs into slices (csrc/pb_slices.h), built for the
host: every pair in one slice, in order, no slice past its limit unless it is
one pair, and so no slice whose elements pass 32 bits, also where the batch's
residues do."""
import ctypes
import os
import random
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(__file__)
CSRC = os.path.join(HERE, "..", "parasail_b200", "csrc")
SOURCE = """
#include "pb_slices.h"
extern "C" long long limit(void) { return CIGAR_SLICE; }
extern "C" int slice_end(const int64_t *o, const int *q, const int *t, int n, int k0, long long limit)
{ return cigar_slice_end(o, q, t, n, k0, limit); }
"""


@pytest.fixture(scope="module")
def slices(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("slices")
    (d / "slices.cpp").write_text(SOURCE)
    so = str(d / "libslices.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "slices.cpp")])
    lib = ctypes.CDLL(so)
    lib.limit.restype = ctypes.c_longlong
    lib.slice_end.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 2 + [ctypes.c_longlong]
    return lib


def _cover(lib, q, t, limit):
    off = np.concatenate([[0], np.cumsum(q[:-1].astype(np.int64) + t[:-1])]).astype(np.int64)
    at, sizes = 0, []
    while at < len(q):
        end = lib.slice_end(off.ctypes.data, q.ctypes.data, t.ctypes.data, len(q), at, limit)
        assert at < end <= len(q)
        size = int(off[end - 1] + q[end - 1] + t[end - 1] - off[at])
        assert size <= limit or end == at + 1
        if end < len(q):
            assert size + int(q[end]) + int(t[end]) > limit      # as few slices as the order allows
        sizes.append(size)
        at = end
    assert sum(sizes) == int(q.astype(np.int64).sum() + t.astype(np.int64).sum())
    return sizes


@pytest.mark.parametrize("n,hi,limit", [(1, 50, 10), (400, 50, 1), (400, 50, 99), (400, 50, 1000), (400, 50, 10 ** 6)])
def test_slices_cover_a_batch(slices, n, hi, limit):
    rng = random.Random(n + limit)
    q, t = (np.array([rng.randint(1, hi) for _ in range(n)], np.int32) for _ in range(2))
    _cover(slices, q, t, limit)


def test_slices_of_a_batch_past_32_bits(slices):
    """200,000 pairs of 30,000 residues each: 1.2e10 elements at most."""
    q = np.full(200000, 30000, np.int32)
    sizes = _cover(slices, q, q, slices.limit())
    assert len(sizes) > 100 and max(sizes) < 2 ** 31 and sum(sizes) > 2 ** 33
