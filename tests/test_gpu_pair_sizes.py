"""Pair batches at the sizes where the int16x2 pair kernels change: rows at
the edges of strips (16) and passes (32), columns at the edges of the four
that run together, the biased and the unbiased form (a penalty that takes
score + open out of int8), alphabets of a few and of many letters, and one
query shared by a task. Every record against the oracle."""
import random
import re

import numpy as np
import pytest

import oracle as O
from conftest import AA, DNA, rand_seq, mutate

pb = pytest.importorskip("parasail_b200")
pytestmark = pytest.mark.gpu

EDGES = (1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 96, 97, 130)
FUNCS = ("nw_striped_32", "nw_stats_striped_32", "sg_striped_32", "sg_qx_stats_scan_32", "sg_dx_striped_32",
         "sg_de_stats_scan_32", "sw_striped_32", "sw_stats_striped_32", "sw_stats_scan_32")


def _check(name, recs, queries, targets, open_, gap, om):
    stats = "_stats" in name
    alg, sgf = O.alg_of(name.split("_striped")[0].split("_scan")[0].replace("_stats", ""))
    keys = ("score", "end_query", "end_ref") + (("matches", "similar", "length") if stats else ())
    for k, (q, t) in enumerate(zip(queries, targets)):
        e = O.align(alg, sgf, int(stats), q, t, open_, gap, om)
        assert tuple(int(recs[k][f]) for f in keys) == tuple(e[f] for f in keys), (name, k, len(q), len(t))


@pytest.mark.parametrize("alphabet,open_,gap", [(DNA, 5, 2), (DNA, 126, 3), (AA, 11, 1), (AA, 120, 2)])
def test_pairs_at_edges(alphabet, open_, gap):
    rng = random.Random(open_ * 10 + gap)
    m = pb.matrix_create("ACGT", 2, -3) if alphabet is DNA else pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    queries, targets = [], []
    for i, a in enumerate(EDGES):
        for b in EDGES[i % 3::3]:
            q = rand_seq(rng, a, alphabet)
            t = (mutate(rng, q, alphabet, 0.1, 0.05) + rand_seq(rng, b, alphabet))[:b] if rng.random() < 0.7 else \
                rand_seq(rng, b, alphabet)
            queries.append(q)
            targets.append(t or rand_seq(rng, b, alphabet))
    for name in FUNCS:
        _check(name, pb.batch_pairs(name, m, queries, targets, open_, gap), queries, targets, open_, gap, om)


@pytest.mark.parametrize("open_,gap", [(11, 1), (120, 2)])
def test_all_against_all_at_edges(open_, gap):
    """Tasks whose pairs share the query."""
    rng = random.Random(open_)
    m = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    seqs = [rand_seq(rng, n, AA) for n in EDGES * 2]
    seqs[7] = mutate(rng, seqs[19], AA, 0.2, 0.05)
    queries = [seqs[i] for i in range(len(seqs)) for j in range(i + 1, len(seqs))]
    targets = [seqs[j] for i in range(len(seqs)) for j in range(i + 1, len(seqs))]
    for name in ("nw_stats_scan_32", "sg_qx_striped_32", "sw_striped_32", "sw_stats_striped_32"):
        _check(name, pb.batch_all(name, m, seqs, open_, gap), queries, targets, open_, gap, om)


@pytest.mark.parametrize("qlen", [1, 2, 31, 33, 64, 65, 300, 1023, 1024, 1025, 2047, 2048, 2049])
def test_single_calls_on_one_block(qlen):
    """One pair per call: queries at the edges of warps, of 2 and 4 rows a
    thread and past the block; every statistic against the oracle, and the
    16-bit forms (whose verdicts read the extremes of the padded rows)
    against the 32-bit ones."""
    rng = random.Random(qlen)
    b62 = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(b62)
    q = rand_seq(rng, qlen, AA)
    targets = [rand_seq(rng, 1, AA), mutate(rng, q, AA, 0.3, 0.05)[:400] or "A", rand_seq(rng, rng.randint(2, 300), AA)]
    prof = pb.ProfileHandle("parasail_profile_create_stats_32", q, b62)
    prof16 = pb.ProfileHandle("parasail_profile_create_stats_16", q, b62)
    for name in ("nw_stats_striped", "sg_qx_stats_scan", "sg_stats_striped", "sw_stats_scan", "nw_scan", "sg_de_striped"):
        stats = "_stats" in name
        alg, sgf = O.alg_of(name.split("_striped")[0].split("_scan")[0].replace("_stats", ""))
        keys = ("score", "end_query", "end_ref") + (("matches", "similar", "length") if stats else ())
        for t in targets:
            e = O.align(alg, sgf, int(stats), q, t, 11, 1, om)
            got = pb.align_profile("parasail_%s_profile_32" % name, prof, t, 11, 1)
            assert all(got[f] == e[f] for f in keys), (name, len(t))
            g16 = pb.align_profile("parasail_%s_profile_16" % name, prof16, t, 11, 1)
            assert not g16["flag"] & pb.FLAG_SATURATED and all(g16[f] == e[f] for f in keys), (name, len(t))


@pytest.mark.parametrize("alg", ["sw", "nw", "sg", "sg_qx", "sg_de"])
def test_batch_cigars_equal_single_ones(alg):
    """CIGARs built on the device against parasail_result_get_cigar on the
    single trace results: mixed case, gaps to the edges, end gaps, pairs of
    one residue, a saturated 8-bit pair."""
    rng = random.Random(len(alg))
    m = pb.matrix_lookup("blosum62")
    qs, ts = ["A", "W", "ARNDW", "W" * 40], ["A", "GGGW", "W", "W" * 40]
    for _ in range(60):
        q = rand_seq(rng, rng.randint(1, 120), AA)
        t = rand_seq(rng, rng.randint(0, 30), AA) + mutate(rng, q, AA, 0.2, 0.1) + rand_seq(rng, rng.randint(0, 30), AA)
        qs.append("".join(c.lower() if rng.random() < 0.3 else c for c in q))
        ts.append("".join(c.lower() if rng.random() < 0.3 else c for c in t) or "A")
    for form in ("", "_striped_8", "_scan_sat"):
        got = pb.batch_pairs_cigar("%s_trace%s" % (alg, form), m, qs, ts, 11, 1)
        for q, t, g in zip(qs, ts, got):
            assert g == pb.trace("parasail_%s_trace%s" % (alg, form), q, t, 11, 1, m), (alg, form, q, t)


@pytest.mark.parametrize("name", ["sw_stats_striped_32", "sw_stats_striped_sat", "sw_stats_scan_32"])
def test_local_statistics_with_pairs_past_16_bits(name):
    """Local statistics in one pass: pairs that the 16-bit kernels take beside
    pairs past their bounds (whose score runs on the exact kernel and whose
    prefix pass follows alone), paths over many blocks and passes, scores of
    0, and ends in the first row and column."""
    rng = random.Random(7)
    m = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    long_a, long_b = rand_seq(rng, 3100, AA), rand_seq(rng, 3050, AA)
    queries = ["W" * 3000, long_a, long_a[:2950], "W", "A", "G" * 40]
    targets = ["W" * 2990, mutate(rng, long_a, AA, 0.5, 0.02), long_b, "W", "W", "W" * 40]
    for _ in range(60):
        q = rand_seq(rng, rng.randint(1, 700), AA)
        queries.append(q)
        targets.append(rand_seq(rng, rng.randint(0, 200), AA) +
                       (mutate(rng, q, AA, 0.4, 0.03) if rng.random() < 0.7 else rand_seq(rng, rng.randint(1, 700), AA)) or "A")
    _check(name, pb.batch_pairs(name, m, queries, targets, 11, 1), queries, targets, 11, 1, om)


def test_batch_cigars_in_several_slices():
    """A batch of more residues than one slice of CIGARs holds (2^26): 400
    pairs over and over, some outside the pair kernels' range, against the 400
    alone."""
    rng = random.Random(26)
    m = pb.matrix_create("ACGT", 100, -100)
    qs, ts = [], []
    for k in range(400):
        q = rand_seq(rng, 700 if k % 50 == 7 else rng.randint(20, 180), DNA)
        qs.append(q)
        ts.append(rand_seq(rng, 10, DNA) + mutate(rng, q, DNA, 0.1, 0.05) + rand_seq(rng, 20, DNA))

    def run(reps):
        qb, qo, ql = pb.pack(qs * reps)
        tb, to, tl = pb.pack(ts * reps)
        n = len(ql)
        rec = np.zeros((n, 8), np.int32)
        out = [np.zeros(int(ql.sum() + tl.sum()), np.uint32)] + [np.zeros(n, np.int32) for _ in range(3)]
        rc = pb.lib.parasail_b200_batch_pairs_cigar(b"sg_trace_striped_32", m, qb.ctypes.data, qo.ctypes.data, ql.ctypes.data,
                                                    tb.ctypes.data, to.ctypes.data, tl.ctypes.data, n, 200, 20,
                                                    rec.ctypes.data, *[x.ctypes.data for x in out])
        assert rc == 0
        return [rec.reshape(reps, -1)] + [x.reshape(reps, -1) for x in out]

    one = run(1)
    assert (one[2] > 0).any() and (one[2] < 0).any()
    reps = 2 ** 26 // one[1].size + 2
    for a, b in zip(run(reps), one):
        assert (a == b).all()


@pytest.mark.parametrize("qlen,tlens", [(1, (1, 31, 32, 33)), (5, (6, 7)), (31, (1, 2)), (513, (1, 8)), (700, (1, 6, 10)),
                                        (1024, (1, 10, 30)), (1500, (1, 4)), (2048, (1, 5, 40))])
def test_single_calls_of_few_cells_or_columns(qlen, tlens):
    """Score-only calls on either side of the lines between one thread, one
    warp and one block, against the oracle; the 16-bit forms read the extremes."""
    rng = random.Random(qlen)
    b62 = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(b62)
    q = rand_seq(rng, qlen, AA)
    prof, prof16 = (pb.ProfileHandle("parasail_profile_create_" + w, q, b62) for w in ("32", "16"))
    for name in ("nw_striped", "sg_scan", "sg_qb_de_striped"):
        alg, sgf = O.alg_of(name.split("_striped")[0].split("_scan")[0])
        for n in tlens:
            t = rand_seq(rng, n, AA)
            e = O.align(alg, sgf, 0, q, t, 11, 1, om)
            for p, w in ((prof, "32"), (prof16, "16")):
                got = pb.align_profile("parasail_%s_profile_%s" % (name, w), p, t, 11, 1)
                assert all(got[k] == e[k] for k in ("score", "end_query", "end_ref")), (name, w, n)


def _read_cigar(cigar, q, t, beg_q, beg_t):
    """[(op, length, start in q, start in t)], the residues under '=' and 'X' compared."""
    runs, i, j = [], beg_q, beg_t
    for n, op in re.findall(r"(\d+)([=XID])", cigar):
        n = int(n)
        if op in "=X":
            assert all((q[i + x] == t[j + x]) == (op == "=") for x in range(n)), (cigar, i, j)
        runs.append((op, n, i, j))
        i += n * (op != "D")
        j += n * (op != "I")
    assert "".join("%d%s" % (n, op) for op, n, _, _ in runs) == cigar
    assert all(a[0] != b[0] for a, b in zip(runs, runs[1:]))
    return runs, i, j


@pytest.mark.parametrize("alg", ["sw", "nw", "sg", "sg_qx", "sg_de", "sg_qb_db"])
@pytest.mark.parametrize("alphabet,open_,gap", [(DNA, 5, 2), (AA, 11, 1), (AA, 120, 2)])
def test_cigars_against_the_oracle(alg, alphabet, open_, gap):
    """CIGARs read back residue by residue: what they consume, their score and
    their counts against the score and the statistics that the oracle gives
    for the path of the same tie rules. Paths over many blocks and passes."""
    rng = random.Random(open_)
    m = pb.matrix_create("ACGT", 2, -3) if alphabet is DNA else pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    a, sgf = O.alg_of(alg)
    qs, ts = ["A", "G" * 40], ["A", "A" * 35]
    for n in EDGES + (200, 333, 512, 600, 1100):
        for _ in range(2):
            q = rand_seq(rng, n, alphabet)
            t = rand_seq(rng, rng.randint(0, 40), alphabet) + mutate(rng, q, alphabet, 0.25, 0.12) + \
                rand_seq(rng, rng.randint(0, 40), alphabet)
            qs.append(q)
            ts.append(t)
    seen = 0
    for q, t, g in zip(qs, ts, pb.batch_pairs_cigar(alg + "_trace", m, qs, ts, open_, gap)):
        e = O.align(a, sgf, 1, q, t, open_, gap, om)
        assert (g["score"], g["end_query"], g["end_ref"]) == (e["score"], e["end_query"], e["end_ref"])
        if alg == "sw" and e["score"] == 0:
            continue
        runs, i, j = _read_cigar(g["cigar"], q, t, g["beg_query"], g["beg_ref"])
        # a path begins with a diagonal step: a gap before it is one to the matrix edge
        lead = runs[0] if runs[0][0] in "ID" else None
        tail = None
        if alg == "sw":
            assert (i, j) == (e["end_query"] + 1, e["end_ref"] + 1)
        else:
            assert (i, j) == (len(q), len(t)) and (g["beg_query"], g["beg_ref"]) == (0, 0)
            if (e["end_query"] + 1, e["end_ref"] + 1) != (len(q), len(t)):
                tail = runs[-1]
                assert tail[2:] == (e["end_query"] + 1, e["end_ref"] + 1) and tail[0] in "ID"
        score = matches = similar = length = 0
        for run in runs:
            op, n, x, y = run
            if op in "ID":
                free = run is tail or (run is lead and (alg == "sw" or sgf & (O.S1_BEG if op == "I" else O.S2_BEG)))
                score -= 0 if free else open_ + (n - 1) * gap
                length += 0 if run is lead or run is tail else n
                continue
            length += n
            for k in range(n):
                s = O.align(O.NW, 0, 0, q[x + k], t[y + k], 10 ** 6, 10 ** 6, om)["score"]
                score += s
                matches += op == "="
                similar += s > 0
        assert (score, matches, similar, length) == (e["score"], e["matches"], e["similar"], e["length"]), (alg, len(q), len(t))
        seen += 1
    assert seen > 40
