"""Phase rounds over slot counts that are no multiple of the batch in which
slots are read, and block sizes whose payload ends in an 8-byte word, starts
off a 16-byte boundary or takes several batches of loads: counts and payload
sums equal the host replay's."""
import pytest

from oracle.phase import PhaseReplay
from tests.helpers import allocator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nslots,n,sizes", [(1, 33, [24]), (2, 1000, [8, 24, 40]),
                                            (3, 4099, [16, 120, 128, 136, 144]),
                                            (4, 513, [256, 264, 1000, 3072])])
def test_phase_rounds_match_replay(torch_cuda, nslots, n, sizes):
    torch = torch_cuda
    seed, thr = 0xBEEF, int(0.9 * 2**32)
    target = int(0.8 * nslots * n)
    want = PhaseReplay(n, nslots, seed, sizes).run(2, thr, thr, target, 64)
    with allocator(memory=512 << 20) as H:
        size_set = torch.tensor(sizes, dtype=torch.int32, device="cuda")
        slots = torch.zeros(nslots * n, dtype=torch.int64, device="cuda")
        slot_sz = torch.zeros(nslots * n, dtype=torch.int32, device="cuda")
        acc = torch.zeros(6, dtype=torch.int64, device="cuda")
        got = H.phase_run(n, nslots, seed, 2, thr, thr, target, size_set, len(sizes), slots,
                          slot_sz, acc)
        assert got["failed"] == 0 and not slots.any().item()
        for k in ("alloc_rounds", "free_rounds", "filled", "mallocs", "frees"):
            assert got[k] == want[k], k
        assert got["written_sum"] == want["wsum"] and got["read_sum"] == want["rsum"]
        st = H.stats()
        assert st["used_chunks"] == 0 and st["status"] == 0


@pytest.mark.parametrize("nslots", [5, 7, 16])
def test_more_slots_than_one_batch(torch_cuda, nslots):
    """Slot counts past the replay's four: every block is counted once, read
    back as written and freed."""
    torch = torch_cuda
    n, sizes = 777, [16, 24, 200]
    with allocator(memory=512 << 20) as H:
        size_set = torch.tensor(sizes, dtype=torch.int32, device="cuda")
        slots = torch.zeros(nslots * n, dtype=torch.int64, device="cuda")
        slot_sz = torch.zeros(nslots * n, dtype=torch.int32, device="cuda")
        acc = torch.zeros(6, dtype=torch.int64, device="cuda")
        for rnd, thr in enumerate((1 << 31, 1 << 31, 0xFFFFFFFF)):
            H.phase_round(0, n, nslots, 5, rnd, thr, slots, slot_sz, acc, size_set, len(sizes))
            torch.cuda.synchronize()
            assert int(acc[0]) == int((slots != 0).sum())
        H.phase_round(1, n, nslots, 5, 9, 1 << 31, slots, slot_sz, acc)
        torch.cuda.synchronize()
        assert int(acc[0]) == int((slots != 0).sum()) > 0
        H.phase_round(1, n, nslots, 5, 10, 0xFFFFFFFF, slots, slot_sz, acc)
        torch.cuda.synchronize()
        a = acc.tolist()
        assert a[0] == 0 and a[1] == 0 and a[2] == a[3] and a[4] == a[5]
        assert not slots.any().item() and H.stats()["used_chunks"] == 0 and H.status() == 0
