"""Edges of the sample and graph kernels that work on vectors: string lengths
around 8-byte words, 16-byte pairs and 24-byte blocks, and into CUDA's heap;
vertex degrees around the doublings, past two half-warp columns and into
CUDA's heap; grids whose lists exceed one walk; counts that are no multiple of a
warp."""
import numpy as np
import pytest

from tests.helpers import allocator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lengths", [
    (1, [0]), (33, [0, 1, 7, 8]), (1000, [7, 8, 9, 15, 16, 17, 22, 23]),
    (4097, [0, 15, 16, 23, 24, 31, 32, 47, 48, 95]), (257, [1000, 1535, 3064, 3071, 3072, 5001])])
def test_string_lengths(torch_cuda, n, lengths):
    import halloc_b200 as H
    torch = torch_cuda
    rng = np.random.default_rng(n)
    la, lb = (rng.choice(lengths, n).astype(np.int32) for _ in range(2))
    # some pairs are compared with another length: one off, and half a word off
    off = rng.choice([0, 0, 1, -1, 8, -8, 4], n)
    want = np.where(la + lb + off < 0, lb, lb + off).astype(np.int32)
    with allocator(memory=512 << 20):
        d = [torch.from_numpy(x).cuda() for x in (la, lb, want)]
        a, b, c = (torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(3))
        cnt = torch.zeros(4, dtype=torch.int64, device="cuda")
        zero = torch.zeros_like(d[0])
        H.strings_alloc(n, d[0], a, cnt)
        H.strings_alloc(n, d[1], b, cnt)
        H.strings_check(n, a, d[0], zero, cnt[1:])
        H.strings_concat(n, c, a, b, cnt)
        H.strings_check(n, c, d[0], d[1], cnt[2:])
        H.strings_check(n, c, d[0], d[2], cnt[3:])
        torch.cuda.synchronize()
        assert cnt.tolist() == [0, 0, 0, int((want != lb).sum())]
        for t in (a, b, c):
            H.strings_free(n, t)
        torch.cuda.synchronize()
        st = H.stats()
        assert st["used_chunks"] == 0 and st["status"] == 0


@pytest.mark.parametrize("n,degrees", [(1, [3]), (31, [0, 1, 2]), (33, [1, 2, 3, 4, 5]),
                                       (1000, [7, 8, 9, 15, 16, 17, 31, 32, 33]),
                                       (200, [0, 63, 64, 65, 511, 512, 513, 1025])])
def test_graph_degrees(torch_cuda, n, degrees):
    import halloc_b200 as H
    from oracle.graph import graph_csr
    torch = torch_cuda
    # thresholds t[k] = share of the hash range with degree <= k
    top = max(degrees)
    share = np.cumsum([degrees.count(k) for k in range(top + 1)]) / len(degrees)
    t = np.minimum(share * 2**32, 2**32 - 1).astype(np.uint32)
    seed = 77
    want_off, want_cols = graph_csr(n, seed, t)
    with allocator(memory=512 << 20):
        cdf = torch.from_numpy(t.view(np.int32)).cuda()
        arr = torch.zeros(n, dtype=torch.int64, device="cuda")
        deg = torch.zeros(n, dtype=torch.int32, device="cuda")
        acc = torch.zeros(3, dtype=torch.int64, device="cuda")
        H.graph_build(n, seed, cdf, len(t), arr, deg, acc)
        torch.cuda.synchronize()
        edges = int(want_off[-1])
        assert acc.tolist()[0] == 0 and acc.tolist()[2] == edges
        off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        off[1:] = torch.cumsum(deg.to(torch.int64), 0)
        cols = torch.full((edges + 16,), -1, dtype=torch.int32, device="cuda")
        H.graph_gather(n, arr, deg, off, cols)
        torch.cuda.synchronize()
        assert np.array_equal(off.cpu().numpy(), want_off)
        got = cols.cpu().numpy()
        assert np.array_equal(got[:edges].view(np.uint32), want_cols) and (got[edges:] == -1).all()
        assert not arr.any().item()
        st = H.stats()
        assert st["used_chunks"] == 0 and st["status"] == 0


@pytest.mark.parametrize("n,ncells", [(1, 1), (31, 1), (129, 1), (2000, 1), (1000, 8), (5001, 3),
                                      (1000, 41), (300000, 41), (999, 64)])
def test_grid_lists(torch_cuda, n, ncells):
    import halloc_b200 as H
    from halloc_b200.workloads import sample_points
    torch = torch_cuda
    with allocator(memory=512 << 20):
        pts = torch.from_numpy(sample_points(n, n)).cuda()
        grid = torch.zeros(ncells**3, dtype=torch.int64, device="cuda")
        count = torch.zeros(ncells**3, dtype=torch.int32, device="cuda")
        hsum = torch.zeros(ncells**3, dtype=torch.int64, device="cuda")
        nfail = torch.zeros(1, dtype=torch.int64, device="cuda")
        for _ in range(2):
            H.grid_insert(n, ncells, pts, grid, nfail)
            H.grid_check(ncells, grid, count, hsum)
            H.grid_free(ncells, grid)
            torch.cuda.synchronize()
            assert int(count.sum()) == n and int(nfail) == 0
            assert not grid.any().item()
            st = H.stats()
            assert st["used_chunks"] == 0 and st["status"] == 0
