"""Caller-supplied device codes outside the alphabet, in queries and targets
of pair batches, read as letter 0 in every kernel: the records equal those of
the same sequences with letter 0 in their place."""
import numpy as np
import pytest

pb = pytest.importorskip("parasail_b200")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def records(name, m, qlens, tlens, open_, gap, outside):
    """Pairs of related random codes, a tenth of them outside the alphabet
    (or letter 0 in the same places)."""
    rng = np.random.RandomState(open_ + len(qlens))
    size = m.contents.size
    sets = []
    text = rng.randint(0, size, int(max(qlens.max(), tlens.max())) + 50).astype(np.uint8)
    for lens in (qlens, tlens):
        offs = np.concatenate([[0], np.cumsum(lens[:-1], dtype=np.int64)]).astype(np.int64)
        codes = np.concatenate([text[:n] for n in lens])
        change = rng.rand(len(codes)) < 0.1
        codes[change] = rng.randint(0, size, int(change.sum()))
        at = rng.randint(0, len(codes), len(codes) // 10 + 1)
        bad = rng.choice([size, size + 1, 31, 32, 128, 254, 255], len(at)).astype(np.uint8)
        codes[at] = bad if outside else 0
        sets += [torch.from_numpy(x).cuda() for x in (codes, offs, lens.astype(np.int32))]
    rec = torch.zeros((len(qlens), 8), dtype=torch.int32, device="cuda")
    rc = pb.lib.parasail_b200_batch_pairs_device(name.encode(), m, *[x.data_ptr() for x in sets], len(qlens), open_, gap,
                                                 rec.data_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    return rec.cpu().numpy()


@pytest.mark.parametrize("name", ["sw_stats_scan_32", "nw_striped_32", "sg_stats_striped_32"])
@pytest.mark.parametrize("rows", [(1, 8), (8, 32), (40, 300)])
def test_exact_kernels(name, rows):
    """Scores past 16 bits: a thread or a warp per pair."""
    rng = np.random.RandomState(rows[0])
    m = pb.matrix_create("ACGT", 3000, -4000)
    q, t = rng.randint(rows[0], rows[1], 70), rng.randint(1, 200, 70)
    a, b = (records(name, m, q, t, 9000, 700, outside) for outside in (False, True))
    assert np.array_equal(a, b)


@pytest.mark.parametrize("name", ["sw_striped_32", "sw_stats_striped_32", "sw_stats_scan_32", "nw_stats_striped_32",
                                  "sg_qx_stats_scan_32", "nw_scan_16"])
@pytest.mark.parametrize("alphabet", ["ACGT", "ARNDCQEGHILKMFPSTWYV"])
def test_pair_kernels(name, alphabet):
    """Scores inside 16 bits: the pair kernels and their traceback."""
    rng = np.random.RandomState(len(alphabet))
    m = pb.matrix_create(alphabet, 2, -3)
    q, t = rng.randint(1, 300, 300), rng.randint(1, 300, 300)
    a, b = (records(name, m, q, t, 5, 2, outside) for outside in (False, True))
    assert np.array_equal(a, b)
