"""The lanes of a warp share the allocations and frees of its jobs: launch
shapes from one warp to full blocks (and both depths of the list walk),
requests above 32 blocks a step, the smallest and the largest block, one job
alone.  Every job's block count and value sum equal those of the default
launch and, for the sums, the host's."""
import numpy as np
import pytest

from tests.helpers import allocator
from tests.test_gpu_serve import value_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,block_bytes,grow_max", [(1, 256, 32), (700, 16, 45), (900, 256, 1),
                                                    (500, 3072, 100)])
def test_launch_shapes_give_one_result(torch_cuda, n, block_bytes, grow_max):
    import halloc_b200 as H
    torch = torch_cuda
    cfg = dict(lam=2e6, seed=5, mean_life=12.0, min_len=64, max_len=48 << 10,
               block_bytes=block_bytes, grow_max=grow_max)
    want = None
    with allocator(memory=2 << 30):
        for threads, per_sm in ((256, 1), (32, 1), (1024, 1), (512, 0), (544, 1)):
            res = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
            r = H.serve_run(res, n, cta_threads=threads, ctas_per_sm=per_sm, **cfg)
            assert r["jobs_done"] == n and r["alloc_failures"] == 0 and r["timeouts"] == 0
            assert int(r["hist"].sum()) == r["allocs"]
            got = res.view(-1, 2).cpu().numpy().astype(np.uint64)
            assert int(got[:, 0].sum()) == r["allocs"]
            if want is None:
                want = got
                assert np.array_equal(got[:, 1], value_sums(np.arange(n), got[:, 0]))
            assert np.array_equal(got, want), (threads, per_sm)
            st = H.stats()
            assert st["used_chunks"] == 0 and st["status"] == 0
