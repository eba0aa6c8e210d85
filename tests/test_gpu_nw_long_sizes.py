"""Global scores of long pairs at the sizes where the int16x2 wavefront
changes: rows at the edges of strips, lanes and passes, targets shorter than
the skew of a warp and at the edges of 32-column chunks, pairs of one warp
and of teams, and the 32-bit wavefront for scores whose steps do not fit 16
bits. Every score against the oracle."""
import random

import numpy as np
import pytest

import oracle as O
from conftest import AA, DNA, rand_seq, mutate

pb = pytest.importorskip("parasail_b200")
pytestmark = pytest.mark.gpu


def _check(m, queries, targets, open_, gap):
    om = O.Matrix.from_struct(m)
    qb, qo, ql = pb.pack(queries)
    tb, to, tl = pb.pack(targets)
    got = pb.nw_long(m, qb, qo, ql, tb, to, tl, open_, gap)
    exp = np.array([O.align(O.NW, 0, 0, q, t, open_, gap, om)["score"] for q, t in zip(queries, targets)], np.int32)
    bad = np.nonzero(got != exp)[0]
    assert len(bad) == 0, [(len(queries[k]), len(targets[k]), int(got[k]), int(exp[k])) for k in bad[:5]]


@pytest.mark.parametrize("alphabet,match,mismatch,open_,gap", [(DNA, 1, -2, 4, 1), (DNA, 2, -3, 5, 5), (AA, 0, 0, 11, 1),
                                                               (AA, 0, 0, 60, 2)])
def test_nw_long_edges(alphabet, match, mismatch, open_, gap):
    rng = random.Random(open_)
    m = pb.matrix_create("ACGT", match, mismatch) if alphabet is DNA else pb.matrix_lookup("blosum62")
    rows = (1, 4, 5, 8, 9, 15, 16, 17, 255, 256, 257, 511, 512, 513, 1023, 1025, 1600)
    cols = (1, 2, 31, 32, 33, 62, 63, 64, 65, 95, 96, 97, 500)
    queries, targets = [], []
    for k, a in enumerate(rows):
        for b in cols[k % 2::2]:
            q = rand_seq(rng, a, alphabet)
            t = mutate(rng, q, alphabet, 0.1, 0.05) if b == 500 else rand_seq(rng, b, alphabet)
            queries.append(q)
            targets.append(t or rand_seq(rng, b, alphabet))
    _check(m, queries, targets, open_, gap)                    # one warp each, and teams for the largest
    for k in (0, len(queries) // 2, len(queries) - 1):
        _check(m, queries[k:k + 1], targets[k:k + 1], open_, gap)


def test_nw_long_drift():
    """Scores far outside 16 bits in both directions, teams of several
    blocks, and a set of unequal pairs."""
    rng = random.Random(5)
    m = pb.matrix_create("ACGT", 3, -4)
    a = rand_seq(rng, 15000, DNA)
    pairs = [(a, a), (a, mutate(rng, a, DNA, 0.1, 0.02)), ("A" * 14000, "C" * 15000), (a, rand_seq(rng, 40, DNA)),
             (rand_seq(rng, 30, DNA), a)]
    _check(m, [p[0] for p in pairs], [p[1] for p in pairs], 8, 2)
    pairs += [(rand_seq(rng, rng.randint(1, 900), DNA), rand_seq(rng, rng.randint(1, 900), DNA)) for _ in range(300)]
    _check(m, [p[0] for p in pairs], [p[1] for p in pairs], 8, 2)


@pytest.mark.parametrize("alphabet,open_,gap", [(DNA, 5, 2), (AA, 11, 1)])
def test_bands_of_long_pairs(alphabet, open_, gap):
    """Bands over many passes: narrow ones that a lane leaves between two
    checks of the base, ones as wide as a pass, scores outside 16 bits, and
    targets much shorter and longer than the query."""
    rng = random.Random(gap)
    m = pb.matrix_create("ACGT", 2, -3) if alphabet is DNA else pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    queries, targets = [], []
    for n in (254, 256, 258, 1300, 2047, 6000):
        q = rand_seq(rng, n, alphabet)
        queries += [q, q, q]
        targets += [mutate(rng, q, alphabet, 0.1, 0.02), rand_seq(rng, n // 2 + 1, alphabet),
                    q + rand_seq(rng, 300, alphabet)]
    for k in (1, 2, 3, 8, 33, 130, 257, 700):
        got = pb.nw_banded_batch(m, queries, targets, open_, gap, k)
        for q, t, g in zip(queries, targets, got):
            assert g == O.nw_banded(q, t, open_, gap, k, om)["score"], (k, len(q), len(t))


@pytest.mark.parametrize("match,mismatch,open_,gap", [(100, -100, 20, 10), (3, -4, 8, 2)])
def test_passes_read_what_the_pass_before_published(match, mismatch, open_, gap):
    """Pairs of more passes than a team of several blocks has warps, so that
    every ring is written over while the next block reads it: (100, -100) in
    the 32-bit wavefront, (3, -4) in the 16-bit one. Insertions and deletions
    make the lanes of one chunk read the ring at different times."""
    rng = random.Random(match)
    m = pb.matrix_create("ACGT", match, mismatch)
    a = rand_seq(rng, 18700, DNA)
    queries = [a, a[:18500], a[:600], a[:300]]
    targets = [mutate(rng, a, DNA, 0.1, 0.04)[:9000], rand_seq(rng, 7000, DNA), mutate(rng, a[:600], DNA, 0.2, 0.1), a[:90]]
    _check(m, queries, targets, open_, gap)


@pytest.mark.parametrize("match,open_,gap", [(2, 5, 2), (100, 200, 20), (100, 20, 10)])
def test_codes_outside_the_alphabet_read_as_letter_0(match, open_, gap):
    """Caller-supplied device codes of the alphabet's size and more, in
    queries and targets, give the scores of letter 0 there: the 16-bit
    wavefront, and the 32-bit one beside the biased form."""
    torch = pytest.importorskip("torch")
    rng = np.random.RandomState(open_)
    m = pb.matrix_create("ACGT", match, -match)
    size = m.contents.size
    rows = []
    for outside in (False, True):
        rng.seed(open_)
        sets = []
        for lo, hi in ((1, 900), (1, 700)):
            lens = rng.randint(lo, hi, 40).astype(np.int32)
            lens[:2] = (3000, 2600)
            offs = np.concatenate([[0], np.cumsum(lens[:-1], dtype=np.int64)]).astype(np.int64)
            codes = rng.randint(0, 4, int(lens.sum())).astype(np.uint8)
            at = rng.randint(0, len(codes), len(codes) // 10)
            bad = rng.choice([size, size + 1, 31, 32, 33, 128, 255], len(at)).astype(np.uint8)
            codes[at] = bad if outside else 0
            sets += [torch.from_numpy(x).cuda() for x in (codes, offs, lens)]
        rec = torch.zeros((40, 8), dtype=torch.int32, device="cuda")
        mask = pb.lib.parasail_b200_schedule_get()
        pb.lib.parasail_b200_schedule_set(0xffffffff)        # every length to the wavefront
        try:
            rc = pb.lib.parasail_b200_batch_pairs_device(b"nw_striped_32", m, *[x.data_ptr() for x in sets], 40, open_, gap,
                                                         rec.data_ptr())
        finally:
            pb.lib.parasail_b200_schedule_set(mask)
        assert rc == 0
        torch.cuda.synchronize()
        rows.append(rec.cpu().numpy())
    assert np.array_equal(rows[0], rows[1])
