"""Pair batches at the sizes where the int16x2 pair kernels change: rows at
the edges of strips (16) and passes (32), columns at the edges of the four
that run together, the biased and the unbiased form (a penalty that takes
score + open out of int8), alphabets of a few and of many letters, and one
query shared by a task. Every record against the oracle."""
import random

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
