"""The device core run on the CPU by warps in seeded random orders
(tests/hostcore): what holds at every order of the accesses to shared memory is
checked over some hundred orders a case, which a GPU meets only by chance.

The slabs are tiny (64 KiB; 27 blocks of 2 KiB up to the busy threshold), so
that heads change all the time and the pool runs out within a few hundred
allocations.  Every case is deterministic: its orders are drawn from the seeds
0 .. n - 1."""
import numpy as np
import pytest

from tests.hostcore.build import NONE, Core, build

SID = {16: 0, 24: 1, 32: 2, 48: 3, 256: 8, 384: 9, 512: 10, 768: 11, 1024: 12, 1536: 13, 2048: 14}


@pytest.fixture(scope="module")
def core(tmp_path_factory):
    return Core(build(tmp_path_factory.mktemp("hostcore")))


def test_one_lane_alone_gets_the_oracles_addresses(core):
    """The host build is the allocator: a lone lane's results over 4,000 calls
    that run through several heads of each size are the oracle's."""
    import oracle
    from tests.trace_gen import make_trace
    ops = np.asarray(make_trace(n=4000, sizes=[256, 384, 512, 1024, 2048], pfree=0.3, seed=5))
    model = oracle.Model(memory=64 << 20, sb_sz_sh=20)
    want = model.run_ops(ops)
    core.init(model.nsbs, sb_sh=20)
    # the oracle's ops name the allocation to free the same way (-op - 1)
    assert np.array_equal(core.cls, model.state().size_infos)
    (got,) = core.run([ops.reshape(-1, 1)], seed=0, hold=0)
    mallocs = ops > 0
    freed = np.zeros(len(ops), bool)
    freed[-ops[ops < 0] - 1] = True
    held = mallocs & ~freed
    assert core.status == 0 and core.nulls == 0
    assert np.array_equal(got[held, 0], want[held])


STORMS = [(2048, 1), (2048, 4), (256, 1), (256, 8)]


@pytest.mark.parametrize("surge", [0, 1])
@pytest.mark.parametrize("size,lanes", STORMS)
def test_no_null_while_a_slab_is_left(core, size, lanes, surge):
    """8 warps allocate until all but a few blocks of what 4 slabs give up to
    the busy threshold is taken: no request may come away empty, whichever
    warp holds the last slab in its hands just then."""
    nsbs, nwarps, sid = 4, 8, SID[size]
    for seed in range(300):
        core.init(nsbs, surge=surge)
        per_slab = int(core.cls[sid, 7]) // int(core.cls[sid, 3])
        k = (nsbs * per_slab - nwarps * lanes) // (nwarps * lanes)
        res = np.concatenate([r.ravel() for r in
                              core.run([np.full((k, lanes), size)] * nwarps, seed)])
        assert (res >= 0).all(), seed
        assert len(np.unique(res)) == len(res), seed
        assert core.nulls == 0 and core.status == 0, seed


@pytest.mark.parametrize("surge", [0, 1])
@pytest.mark.parametrize("size,lanes", STORMS)
def test_a_null_leaves_no_slab_unused(core, size, lanes, surge):
    """8 warps ask for more than 4 slabs hold: once the last request is
    answered no slab lies prefetched, and every slab is filled to the busy
    threshold but for the blocks that were on their way when it was left."""
    nsbs, nwarps, sid = 4, 8, SID[size]
    for seed in range(300):
        core.init(nsbs, surge=surge)
        ncib, busy = int(core.cls[sid, 3]), int(core.cls[sid, 7])
        k = nsbs * int(core.cls[sid, 0]) // ncib // (nwarps * lanes) + 1
        core.run([np.full((k, lanes), size)] * nwarps, seed)
        assert core.nulls > 0 and core.status == 0, seed
        assert core.head(sid)["prefetched"] == NONE, seed
        used = [core.slab(sb)["used"] for sb in range(nsbs)]
        assert min(used) >= busy - nwarps * lanes * ncib, (seed, used)
