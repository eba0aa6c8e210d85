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


@pytest.mark.parametrize("open_,gap", [(11, 1), (120, 2)])
def test_few_pairs_wavefront(open_, gap):
    """Small searches and single calls: queries at the edges of the rows a
    lane and a pass hold, targets of one residue and more; (120, 2) is past
    the biased form. Every pair against the oracle."""
    rng = random.Random(open_)
    b62 = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(b62)
    lengths = [1, 2, 63, 64, 65, 127, 128, 129, 191, 193, 300, 319, 320, 321, 385, 448, 512, 513, 577, 1100]
    for k, L in enumerate(lengths):
        q = rand_seq(rng, L, AA)
        targets = [rand_seq(rng, 1, AA), rand_seq(rng, 2, AA), q, mutate(rng, q, AA, 0.3, 0.05) + rand_seq(rng, 40, AA)]
        targets += [rand_seq(rng, rng.randint(1, 700), AA) for _ in range(3)]
        prof = pb.ProfileHandle("parasail_profile_create_16", q, b62)
        recs = pb.batch_profile("sw_striped_profile_16", prof, targets, open_, gap)
        for i, t in enumerate(targets):
            e = O.align(O.SW, 0, 0, q, t, open_, gap, om)
            exp = (e["score"], e["end_query"], e["end_ref"])
            assert tuple(int(recs[i][f]) for f in FIELDS[:3]) == exp, (L, i)
            got = pb.align_profile("parasail_sw_striped_profile_16", prof, t, open_, gap)
            assert (got["score"], got["end_query"], got["end_ref"]) == exp, (L, i)
        prof.close()
    queries = [rand_seq(rng, L, AA) for L in (40, 300, 700)]
    _check_db(queries, [rand_seq(rng, rng.randint(1, 500), AA) for _ in range(130)], "sw_striped_profile_16",
              open_, gap, 130, 3)


@pytest.mark.parametrize("qlens,n", [((300,), 40), ((300,), 12000), ((60, 700, 1500), 5000), ((2000,), 10000)])
def test_codes_outside_the_alphabet_read_as_letter_0(qlens, n):
    """Caller-supplied device codes of the alphabet's size and more give the
    records of the same targets with letter 0 there, whatever kernel the size
    selects (the few-pairs kernel, warps, teams), also from a plan."""
    torch = pytest.importorskip("torch")
    rng = np.random.RandomState(n)
    b62 = pb.matrix_lookup("blosum62")
    size = b62.contents.size
    lens = rng.randint(1, 400, n).astype(np.int32)
    offs = np.concatenate([[0], np.cumsum(lens[:-1], dtype=np.int64)]).astype(np.int64)
    codes = rng.randint(0, size, int(lens.sum())).astype(np.uint8)
    at = rng.randint(0, len(codes), len(codes) // 20)
    codes[at] = rng.choice([size, size + 1, 31, 32, 127, 128, 200, 255], len(at)).astype(np.uint8)
    clean = np.where(codes < size, codes, 0).astype(np.uint8)
    profs = [pb.ProfileHandle("parasail_profile_create_sat", rand_seq(random.Random(L), L, AA), b62) for L in qlens]
    parr = pb.ctypes.cast(pb.profile_array(profs), pb.ctypes.c_void_p)
    d_offs, d_lens = torch.from_numpy(offs).cuda(), torch.from_numpy(lens).cuda()
    recs = []
    for c in (clean, codes):
        d_codes = torch.from_numpy(c).cuda()
        for plan in (False, True):
            rec = torch.zeros((len(qlens), n, 8), dtype=torch.int32, device="cuda")
            args = (b"sw_striped_profile_sat", parr, len(qlens), d_codes.data_ptr(), d_offs.data_ptr(), d_lens.data_ptr(),
                    n, 11, 1, rec.data_ptr())
            if plan:
                h = pb.lib.parasail_b200_db_plan_create(*args)
                assert h and pb.lib.parasail_b200_db_plan_run(h) == 0
                pb.lib.parasail_b200_db_plan_free(h)
            else:
                assert pb.lib.parasail_b200_batch_db_device(*args) == 0
            torch.cuda.synchronize()
            recs.append(rec.cpu().numpy())
    for r in recs[1:]:
        assert np.array_equal(r, recs[0])
