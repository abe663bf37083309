"""Tickets under surge head sets: which counter a warp draws from is told by a
cached copy of the size's level, which may be stale.  Storms that open levels,
levels closed between launches, and threads alone in their warps beside full
warps: checksums, counts and the empty pool stay exact."""
import pytest

from tests.helpers import allocator, assert_free_count, plain_checksum

pytestmark = pytest.mark.gpu


def run(torch, H, n, nbytes, nallocs, niters, block):
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    H.throughput(out, n, nbytes=nbytes, block=block, nallocs=nallocs, niters=niters)
    torch.cuda.synchronize()
    return out.cpu().tolist()


@pytest.mark.parametrize("nbytes,n,nallocs", [(16, 1 << 20, 2), (256, 1 << 20, 1),
                                              (768, 200003, 1), (3072, 65537, 1)])
def test_levels_opened_and_closed_between_launches(torch_cuda, nbytes, n, nallocs):
    torch = torch_cuda
    with allocator(memory=1 << 30) as H:
        levels = []
        for rep in range(6):
            assert run(torch, H, n, nbytes, nallocs, 2, 128) == [plain_checksum(n, 2 * nallocs), 0]
            levels.append(max(H.stats()["surge_level"]))
            if rep % 2:
                H.close_surges()
            # a few warps, and warps of one thread, against whatever is open
            assert run(torch, H, 97, nbytes, 1, 3, 32) == [plain_checksum(97, 3), 0]
            assert run(torch, H, 200, nbytes, 1, 2, 1) == [plain_checksum(200, 2), 0]
        st = H.stats()
        assert nbytes == 16 or max(levels) > 0, levels
        assert st["used_chunks"] == 0 and H.status() == 0
        assert_free_count(H)
