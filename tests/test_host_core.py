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


def churn(rng, nops, lanes, sizes, p_free, keep=0.0):
    """A warp's random allocations and frees; what it holds at the end it frees
    but for the share `keep`."""
    ops, held = [], []
    for _ in range(nops):
        if held and rng.random() < p_free:
            ops.append([-held.pop(rng.integers(len(held))) - 1] * lanes)
        else:
            held.append(len(ops))
            ops.append(list(rng.choice(sizes, lanes)))
    ops += [[-k - 1] * lanes for k in held if rng.random() >= keep]
    return np.array(ops)


def assert_quiescent(core, res, seed):
    """No block handed out twice, the counts those of the blocks held, and every
    slab where it belongs: a head, a prefetched slab or in a set."""
    held = np.concatenate([r[r >= 0] for r in res])
    assert len(np.unique(held)) == len(held), seed
    owned = {core.head(s, k)[w] for s in range(16) for k in range(16)
             for w in ("slab", "prefetched")}
    for sb in range(core.nsbs):
        d = core.slab(sb)
        blocks = int(((held >> core.sb_sh) == sb).sum())
        ncib = int(core.cls[d["size_id"], 3]) if d["size_id"] != NONE else 0
        assert d["is_head"] == d["head_flag"] == (sb in owned), (seed, sb, d)
        assert (d["used"] == 0) == (blocks == 0), (seed, sb, d)
        if d["is_head"] or d["size_id"] == NONE:
            continue
        # A head that is detached with exactly its busy threshold in use is in no
        # set until it is roomy (the reference's rule); blocks of several chunks
        # never add up to a threshold that is odd.
        busy = int(core.cls[d["size_id"], 7])
        if ncib > 1 and busy % 2 and d["used"] < busy:
            assert d["nsets"] > 0, (seed, sb, d)


@pytest.mark.parametrize("surge", [0, 1])
@pytest.mark.parametrize("sizes,lanes", [([2048], 1), ([2048], 4), ([1024, 2048], 2),
                                         ([512, 768, 2048], 4)])
def test_a_slab_with_room_is_in_a_set(core, sizes, lanes, surge):
    """Warps allocate and free at random and hold half of what they have at the
    end: frees race the changes of the heads that they free into."""
    for seed in range(250):
        rng = np.random.default_rng(seed)
        core.init(int(rng.integers(4, 16)), surge=surge)
        res = core.run([churn(rng, int(rng.integers(20, 120)), lanes, sizes, 0.4, 0.5)
                        for _ in range(int(rng.integers(2, 12)))], seed)
        assert core.status == 0, seed
        assert_quiescent(core, res, seed)


@pytest.mark.parametrize("sizes,lanes", [([2048], 4), ([256], 8), ([512, 768, 2048], 4)])
def test_a_level_changes_only_where_it_is_judged(core, sizes, lanes):
    """Warps storm sizes whose levels open and close: every change of the level
    in a head word is one that was decided (and counted), and the copy of the
    level beside it is right once the warps are done."""
    moves = 0
    for seed in range(250):
        rng = np.random.default_rng(seed)
        core.init(int(rng.integers(6, 40)))
        core.run([churn(rng, int(rng.integers(20, 120)), lanes, sizes, rng.uniform(0.1, 0.5), 0.5)
                  for _ in range(int(rng.integers(2, 12)))], seed)
        assert core.status == 0 and core.level_moves == core.surge_changes, seed
        for size in sizes:
            h = core.head(SID[size])
            assert h["level"] == h["level_copy"], (seed, size, h)
        moves += core.level_moves
    assert moves > 0


@pytest.mark.parametrize("sb_sh", [16, 20, 21, 22, 23, 24])
@pytest.mark.parametrize("fractions", [{}, {"busy": 0.91, "roomy": 0.5, "sparse": 0.0125}])
def test_a_free_sees_the_thresholds_of_every_size_of_the_chunk(core, sb_sh, fractions):
    """A slab's size may change, within its chunk size, between a free's reading
    of the descriptor and the lowering of its count: whichever size it read,
    the free has to notice that it takes the slab over a threshold."""
    core.init(4, sb_sh=sb_sh, **fractions)
    c = core.cls.astype(int)
    for now in range(16):
        for seen in (s for s in range(16) if c[s, 2] == c[now, 2]):
            for t in c[now, [4, 6, 7]]:
                for n in sorted({1, 2, 3, c[now, 3], 8 * c[now, 3], 32 * c[now, 3]}):
                    for n0 in range(t + 1, min(t + n, c[now, 0]) + 1):
                        if n0 >= n:
                            assert core.lib.hc_crosses(int(seen), n0, int(n)), (now, seen, t, n0, n)


@pytest.mark.parametrize("sb_sh", [20, 22, 24])
def test_the_topmost_level_opens_by_pool_and_head_size(core, sb_sh):
    """Levels 1 to 3 need a quarter of the pool free; level 4 a pool of 160 slabs
    with half of them free, or three eighths where a head holds fewer than 4,096
    blocks, which depends on the size and on the slabs."""
    core.init(4, sb_sh=sb_sh)
    room = core.lib.hc_room
    for sid in range(16):
        blocks = int(core.cls[sid, 0]) // int(core.cls[sid, 3])
        for committed in (159, 160, 192, 1000):
            for level in (1, 3, 4, 5):
                for nfree in range(committed + 1):
                    want = 4 * nfree >= committed
                    if level >= 4:
                        eighths = 3 if blocks < 4096 else 4
                        want = level == 4 and committed >= 160 and 8 * nfree >= eighths * committed
                    assert bool(room(sid, level, nfree, committed)) == want, (sid, level, nfree)
