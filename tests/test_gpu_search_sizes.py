"""Database searches over the sizes at which the Smith-Waterman score path
changes its kernel or its split of the work: more queries than fit the
shared memory of the few-pairs kernel, few and many targets, teams and
single warps, and pairs past the 16-bit range among them."""
import random

import numpy as np
import pytest

import oracle as O
from conftest import AA, rand_seq, mutate

pb = pytest.importorskip("parasail_b200")
pytestmark = pytest.mark.gpu

FIELDS = ("score", "end_query", "end_ref", "flag")


def _check_db(queries, targets, name, open_, gap, sample, seed):
    """batch_db against one batch_profile per query, every record, and a
    sample of the pairs against the oracle."""
    b62 = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(b62)
    profs = [pb.ProfileHandle("parasail_profile_create_" + name.rsplit("_", 1)[1], q, b62) for q in queries]
    recs = pb.batch_db(name, profs, targets, open_, gap)
    for q, p in enumerate(profs):
        one = pb.batch_profile(name, p, targets, open_, gap)
        for f in FIELDS:
            assert np.array_equal(recs[q][f], one[f]), (name, q, f)
    rng = random.Random(seed)
    for _ in range(sample):
        q, t = rng.randrange(len(queries)), rng.randrange(len(targets))
        if recs[q][t]["flag"] & pb.FLAG_SATURATED:
            continue
        e = O.align(O.SW, 0, 0, queries[q], targets[t], open_, gap, om)
        got = tuple(int(recs[q][t][f]) for f in FIELDS[:3])
        assert got == (e["score"], e["end_query"], e["end_ref"]), (name, q, t)


@pytest.mark.parametrize("n_targets,t_hi", [(3, 400), (300, 400), (12000, 60)])
def test_many_queries(n_targets, t_hi):
    rng = random.Random(n_targets)
    queries = [rand_seq(rng, L, AA) for L in (1, 31, 32, 33, 500, 777, 1000, 1500, 2000, 2500, 2990, 64)]
    queries[10] = "W" * 2990
    targets = [mutate(rng, queries[5][:300], AA, 0.3, 0.03) if k % 50 == 0 else rand_seq(rng, rng.randint(1, t_hi), AA)
               for k in range(n_targets)]
    targets[1] = "W" * 2995        # 32890 against the query of 2990: past 16 bits
    _check_db(queries, targets, "sw_striped_profile_sat", 11, 1, 60, 1)
    _check_db(queries[4:9] + queries, targets, "sw_scan_profile_32", 10, 2, 20, 2)
