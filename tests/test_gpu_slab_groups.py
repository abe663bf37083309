"""Warp-aggregated counts of slabs that hold blocks of two sizes: lanes of one
warp that free a slab's blocks of different lengths in chunks are counted in
groups of their own, and a free in a slab that is no head files it whenever a
threshold is crossed."""
import numpy as np
import pytest

from tests.helpers import allocator, assert_free_count, check_blocks
from tests.test_gpu_concurrent import assert_empty, assert_state_matches_live, malloc_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b", [(16, 32), (16, 128), (24, 192), (384, 768)])
def test_frees_in_a_slab_of_two_sizes(torch_cuda, a, b):
    torch = torch_cuda
    with allocator(memory=512 << 20, sb_sz_sh=20, sparse_fraction=0.05) as H:
        st = H.stats()
        chunk = a
        per_slab = (1 << 20) // chunk
        n = 3 * per_slab
        sizes_a = np.full(n, a, np.int64)
        ptrs = malloc_batch(torch, H, sizes_a, n, 1).cpu().numpy()
        check_blocks(ptrs, sizes_a, st["pool_base"], st["pool_bytes"])
        # leave 3 % of every slab: no head any more, filed as sparse
        keep = np.zeros(n, bool)
        slab = (ptrs - st["pool_base"]) >> 20
        for s in np.unique(slab):
            keep[np.flatnonzero(slab == s)[: per_slab * 3 // 100]] = True
        H.free_batch(torch.tensor(np.where(keep, 0, ptrs), device="cuda"), n, 1)
        torch.cuda.synchronize()
        rest = ptrs[keep]
        assert_state_matches_live(H, rest, np.full(len(rest), a, np.int64))
        # blocks of the longer size go into the sparse slabs
        m = len(rest)
        sizes_b = np.full(m, b, np.int64)
        q = malloc_batch(torch, H, sizes_b, m, 1).cpu().numpy()
        assert np.intersect1d((q - st["pool_base"]) >> 20, (rest - st["pool_base"]) >> 20).size
        both = np.stack([rest, q], 1).reshape(-1)  # the two sizes in every warp
        sizes = np.tile([a, b], m)
        check_blocks(both, sizes, st["pool_base"], st["pool_bytes"])
        assert_state_matches_live(H, both, sizes)
        H.free_batch(torch.tensor(both, device="cuda"), 2 * m, 1)
        torch.cuda.synchronize()
        assert_empty(H)
        end = assert_free_count(H)
        assert end["free_slabs"] + end["head_slabs"] == st["nsbs"]
        assert H.status() == 0
