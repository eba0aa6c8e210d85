"""What the library takes of the device's and the host's memory."""
import numpy as np
import pytest

pb = pytest.importorskip("parasail_b200")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _reads(n, seed):
    """n reads of 100 to 300 and their windows as device codes."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ql = torch.randint(100, 301, (n,), generator=g, device="cuda")
    tl = ql + 32
    text = torch.randint(0, 4, (int(tl.sum()),), generator=g, device="cuda").to(torch.uint8)
    toff = torch.cumsum(tl, 0) - tl
    return text, toff, ql.int(), tl.int()       # a read: the first residues of its window


def test_checkpoints_leave_half_of_the_free_memory():
    """A batch whose checkpoints (20 GB) do not fit the free memory takes at
    most half of it, and gives the records that it gives with room enough."""
    n = 1000000
    m = pb.matrix_create("ACGT", 2, -3)
    text, off, ql, tl = _reads(n, 3)
    rec = [torch.zeros((n, 8), dtype=torch.int32, device="cuda") for _ in range(2)]

    def run(out):
        rc = pb.lib.parasail_b200_batch_pairs_device(b"nw_stats_striped_32", m, text.data_ptr(), off.data_ptr(), ql.data_ptr(),
                                                     text.data_ptr(), off.data_ptr(), tl.data_ptr(), n, 5, 2, out.data_ptr())
        assert rc == 0
        torch.cuda.synchronize()

    free = torch.cuda.mem_get_info()[0]
    left = 12 << 30
    assert free > 2 * left
    hold = torch.empty(free - left, dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    run(rec[0])
    after = torch.cuda.mem_get_info()[0]
    del hold
    torch.cuda.empty_cache()
    # beside the checkpoints a few words per pair
    assert before - after <= before // 2 + 200 * n, (before, after)
    run(rec[1])
    assert torch.equal(rec[0], rec[1])
    assert int(rec[0][:, 4].min()) > 0


def test_single_calls_pin_one_block_a_thread():
    """Long targets pin no more memory than short ones, threads that end hand
    their block on, and results are right at the sizes around the block's."""
    import ctypes
    import random
    import threading

    import oracle as O
    from conftest import AA, rand_seq

    pinned = pb.lib.pb_single_pinned_bytes
    pinned.restype = ctypes.c_size_t
    rng = random.Random(8)
    m = pb.matrix_lookup("blosum62")
    om = O.Matrix.from_struct(m)
    q = rand_seq(rng, 40, AA)
    sw, nw = (pb.ProfileHandle("parasail_profile_create_" + c, q, m) for c in ("16", "stats_16"))
    block = 64 << 10
    text = rand_seq(rng, 200000, AA)

    def check(n):
        t = text[-n:]
        e = O.align(O.SW, 0, 0, q, t, 11, 1, om)
        got = pb.align_profile("parasail_sw_striped_profile_16", sw, t, 11, 1)
        assert (got["score"], got["end_query"], got["end_ref"]) == (e["score"], e["end_query"], e["end_ref"]), n
        alg, sgf = O.alg_of("sg")
        e = O.align(alg, sgf, 1, q, t, 11, 1, om)
        got = pb.align_profile("parasail_sg_stats_striped_profile_16", nw, t, 11, 1)
        assert all(got[k] == e[k] for k in e), n

    check(300)
    base = pinned()
    assert base >= block
    for n in [block - d for d in (1000, 600, 400, 350, 300, 256, 200, 100, 1, 0)] + [block + 1, 200000, 10]:
        check(n)
    assert pinned() == base
    wrong = []

    def run(n):
        try:
            check(n)
        except BaseException as e:
            wrong.append(e)

    for _ in range(20):                            # one after the other: one block for all of them
        th = threading.Thread(target=run, args=(200,))
        th.start()
        th.join()
    assert pinned() <= base + block
    ths = [threading.Thread(target=run, args=(1000 + k,)) for k in range(6)]
    for th in ths:
        th.start()
    for th in ths:
        th.join()
    assert not wrong
    assert pinned() <= base + 6 * block
    for p in (sw, nw):
        p.close()
