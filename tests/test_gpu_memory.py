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
