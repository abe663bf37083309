"""Performance cases: the allocator's workloads through the package's public
entry points, from a few microseconds of small calls to the largest runs of
the benchmark.

Every case is one pass of device work that allocates, uses and frees its
blocks, so the pool is empty again after it.  A process runs one case after
another; each case gets a freshly initialised pool (its states share it, as
the calls of one program do).  Addresses differ from run to run under
concurrency, so the outputs are what the blocks held and what the workloads
counted: whole numbers that depend on the inputs alone.
"""
import math

import numpy as np
import torch

import halloc_b200 as H
from halloc_b200.workloads import (BatchedRunner, batched_plan, group_seeds, poisson_thresholds,
                                   sample_lengths, sample_points)

MIB = 1 << 20
THR95 = int(0.95 * 2**32)
PHASE_SIZES = [16, 24, 32, 48, 64, 96, 128, 192, 256]
# bit-array words of one malloc/free pair: one read and written by each side
META = 16


def listed():
    return [
        # the smallest calls: a thousand list nodes into a small grid, one
        # launch each to insert, walk and free
        {"name": "grid_1k", "kind": "grid", "n": 1000, "ncells": 8, "pool_mib": 512},
        # the grid-points sample at its own size: 1 M nodes, 32 per cell
        {"name": "grid_1M", "kind": "grid", "n": 1 << 20, "ncells": 32, "pool_mib": 512},
        # the add-strings sample: 1 M pairs of strings of 0 to 31 characters
        {"name": "strings_1M", "kind": "strings", "n": 1 << 20, "lo": 0, "hi": 31,
         "period": 32, "pool_mib": 512},
        # random-graph build with doubling arrays, then the CSR gather
        {"name": "graph_1M", "kind": "graph", "n": 1 << 20, "degree": 16, "pool_mib": 1024},
        # the plain private loop: 32 K threads, one 16-byte block each, ten times
        {"name": "plain_32k", "kind": "loop", "n": 1 << 15, "nallocs": 1, "niters": 10,
         "lo": 16, "hi": 16, "pool_mib": 512},
        # mixed sizes over the whole range of the slabs, an odd thread count,
        # three blocks held at a time
        {"name": "loop_mixed", "kind": "loop", "n": 20011, "nallocs": 3, "niters": 4,
         "lo": 1, "hi": 3072, "pool_mib": 1024},
        # mixed-size phases with payload: slots filled to 91 %, then mostly freed
        {"name": "phase_1M", "kind": "phase", "n": 1 << 20, "nslots": 4, "periods": 2,
         "pool_mib": 1024},
        # halloc's phase experiment, one launch per try: 256-byte blocks from
        # a million threads (one alloc or free each per launch)
        {"name": "spree_256_1M", "kind": "ref", "n": 1 << 20, "nallocs": 1, "niters": 1,
         "ntries": 8, "smin": 256, "smax": 256, "pool_mib": 512},
        # the same experiment over all sizes, every thread a private loop
        {"name": "private_8_3072", "kind": "ref", "n": 1 << 17, "nallocs": 1, "niters": 8,
         "ntries": 2, "smin": 8, "smax": 3072, "pool_mib": 1024},
        # the batched request stream without and with its 1 % of large
        # requests (CUDA's heap serves those), one persistent launch
        {"name": "batched_small", "kind": "batched", "nbatch": 16, "max_batch": 1 << 18,
         "large": 0.0, "pool_mib": 4096},
        {"name": "batched_large", "kind": "batched", "nbatch": 16, "max_batch": 1 << 16,
         "large": 0.01, "pool_mib": 4096},
        # the serving loop: host-fed jobs, continuous batching, 256-byte blocks
        {"name": "serve_100k", "kind": "serve", "n": 100_000, "pool_mib": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "strings", "graph", "loop", "loop", "phase", "ref", "ref",
                       "ref", "batched"])
    if kind == "grid":
        return {"kind": kind, "n": _log(rng, 500, 1 << 20), "ncells": _log(rng, 8, 64),
                "pool_mib": 512}
    if kind == "strings":
        n = _log(rng, 1000, 1 << 20)
        # live at once: 4 strings' worth of the mean length per pair
        hi = max(8, min(_log(rng, 8, 1000), (64 * MIB) // n))
        return {"kind": kind, "n": n, "lo": rng.randrange(0, hi // 2), "hi": hi,
                "period": rng.choice([1, 32]), "pool_mib": 1024}
    if kind == "graph":
        return {"kind": kind, "n": _log(rng, 2000, 1 << 20), "degree": rng.randint(4, 16),
                "pool_mib": 1024}
    if kind == "loop":
        n, nallocs = _log(rng, 32, 1 << 18), rng.randint(1, 4)
        room = min(3072, (160 * MIB) // (n * nallocs))
        lo = min(_log(rng, 8, 3072), room)
        hi = rng.choice([lo, min(room, 4 * lo), room])
        return {"kind": kind, "n": n, "nallocs": nallocs, "niters": rng.randint(1, 10),
                "lo": lo, "hi": hi, "pool_mib": 1024}
    if kind == "phase":
        return {"kind": kind, "n": _log(rng, 4000, 1 << 20), "nslots": rng.randint(1, 4),
                "periods": rng.randint(1, 2), "pool_mib": 1024}
    if kind == "ref":
        n, nallocs = _log(rng, 1000, 1 << 20), rng.choice([1, 1, 2, 4])
        room = min(3072, (160 * MIB) // (n * nallocs))
        smin = min(_log(rng, 8, 3072), room)
        smax = rng.choice([smin, smin, min(room, 8 * smin), room])
        return {"kind": kind, "n": n, "nallocs": nallocs, "niters": rng.choice([1, 2, 4, 8]),
                "ntries": rng.choice([2, 4, 8]), "smin": smin, "smax": smax, "pool_mib": 1024}
    return {"kind": kind, "nbatch": rng.randint(4, 16), "max_batch": _log(rng, 4000, 1 << 17),
            "large": rng.choice([0.0, 0.0, 0.01]), "pool_mib": 4096}


_open = {"case": None, "heap": False}


def _open_pool(case):
    """A fresh pool for each case.  CUDA fixes the size of its own heap at the
    process's first launch, so the first pool has the largest heap that a
    case here needs (2 GiB) and one launch is made with it."""
    key = {k: v for k, v in case.items() if k != "name"}
    if _open["case"] == key:
        return
    if _open["case"] is not None:
        torch.cuda.synchronize()
        H.shutdown()
        _open["case"] = None
    if not _open["heap"]:
        H.init(H.HallocOpts(memory=4096 * MIB, halloc_fraction=0.5))
        H.throughput(torch.zeros(2, dtype=torch.int64, device="cuda"), 32)
        torch.cuda.synchronize()
        H.shutdown()
        _open["heap"] = True
    frac = 0.5 if case["kind"] == "batched" else 0.75
    H.init(H.HallocOpts(memory=case["pool_mib"] * MIB, halloc_fraction=frac))
    _open["case"] = key


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _zeros(n, dtype):
    return torch.zeros(n, dtype=dtype, device="cuda")


def prepare(case, seed):
    _open_pool(case)
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"case": case, "kind": kind}
    if kind == "grid":
        n3 = case["ncells"] ** 3
        s.update(pts=_dev(sample_points(case["n"], seed)), grid=_zeros(n3, torch.int64),
                 count=_zeros(n3, torch.int32), hsum=_zeros(n3, torch.int64),
                 nfail=_zeros(1, torch.int64))
    elif kind == "strings":
        n, p, lo, hi = case["n"], case["period"], case["lo"], case["hi"]
        la, lb = sample_lengths(n, p, lo, hi, 2 * seed), sample_lengths(n, p, lo, hi, 2 * seed + 1)
        # the lengths the results are compared with: those of the
        # concatenation but for a few per cent that expect something else
        want = lb + (rng.random(n) < 0.05) * rng.integers(1, 9, n).astype(np.int32)
        s.update(la=_dev(la), lb=_dev(lb), want=_dev(want.astype(np.int32)),
                 a=_zeros(n, torch.int64), b=_zeros(n, torch.int64), c=_zeros(n, torch.int64),
                 counts=_zeros(2, torch.int64))
    elif kind == "graph":
        n = case["n"]
        cdf = poisson_thresholds(float(case["degree"]))
        # room for the columns: the mean and six standard deviations
        cap = int(n * case["degree"] + 6 * math.sqrt(n * case["degree"])) + 64
        s.update(seed=int(rng.integers(0, 1 << 32)), cdf=_dev(cdf.view(np.int32)),
                 ncdf=len(cdf), arr=_zeros(n, torch.int64), deg=_zeros(n, torch.int32),
                 offsets=_zeros(n + 1, torch.int64), cols=_zeros(cap, torch.int32),
                 acc=_zeros(3, torch.int64))
    elif kind == "loop":
        sizes = rng.integers(case["lo"], case["hi"] + 1, case["n"]).astype(np.int32)
        # the totals go on from where the program's earlier calls left them
        s.update(sizes=_dev(sizes),
                 out=_dev(np.array([rng.integers(0, 1 << 40), 0], np.int64)))
    elif kind == "phase":
        k = case["nslots"] * case["n"]
        s.update(seed=int(rng.integers(0, 1 << 32)), sizes=_dev(np.array(PHASE_SIZES, np.int32)),
                 slots=_zeros(k, torch.int64), slot_sz=_zeros(k, torch.int32),
                 acc=_zeros(6, torch.int64))
    elif kind == "ref":
        n = case["n"]
        s.update(states=_dev(group_seeds(n, 32, seed).view(np.int32)),
                 slots=_zeros(n * case["nallocs"], torch.int64), ctrs=_zeros(n, torch.int32),
                 acc=_zeros(4, torch.int64), probs=H.phase_ref_probabilities(0.95, 0.05, 0.91))
    elif kind == "batched":
        plan = batched_plan(seed=seed, nbatch=case["nbatch"], max_batch=case["max_batch"],
                            large_frac=case["large"])
        s["runner"] = BatchedRunner(plan, torch)
        s["handle"] = s["runner"].prepare(block=1024, task_items=8192, graph=True)
    else:
        s.update(seed=int(rng.integers(0, 1 << 32)), results=_zeros(2 * case["n"], torch.int64))
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "grid":
        s["nfail"].zero_()
        H.grid_insert(case["n"], case["ncells"], s["pts"], s["grid"], s["nfail"])
        H.grid_check(case["ncells"], s["grid"], s["count"], s["hsum"])
        H.grid_free(case["ncells"], s["grid"])
        return {"count": s["count"], "hsum": s["hsum"], "nfail": s["nfail"]}
    if kind == "strings":
        n, c = case["n"], s["counts"]
        c.zero_()
        H.strings_alloc(n, s["la"], s["a"], c)
        H.strings_alloc(n, s["lb"], s["b"], c)
        H.strings_concat(n, s["c"], s["a"], s["b"], c)
        H.strings_check(n, s["c"], s["la"], s["want"], c[1:])
        for t in ("a", "b", "c"):
            H.strings_free(n, s[t])
        return {"failed_and_different": c, "a": s["a"], "b": s["b"], "c": s["c"]}
    if kind == "graph":
        n = case["n"]
        H.graph_build(n, s["seed"], s["cdf"], s["ncdf"], s["arr"], s["deg"], s["acc"])
        torch.cumsum(s["deg"], 0, dtype=torch.int64, out=s["offsets"][1:])
        H.graph_gather(n, s["arr"], s["deg"], s["offsets"], s["cols"])
        return {"cols": s["cols"], "offsets": s["offsets"], "acc": s["acc"]}
    if kind == "loop":
        H.throughput(s["out"], case["n"], nallocs=case["nallocs"], niters=case["niters"],
                     sizes=s["sizes"])
        return s["out"]
    if kind == "phase":
        n = case["n"]
        H.phase_run(n, case["nslots"], s["seed"], case["periods"], THR95, THR95,
                    int(0.91 * case["nslots"] * n), s["sizes"], len(PHASE_SIZES), s["slots"],
                    s["slot_sz"], s["acc"])
        return {"acc": s["acc"], "slots": s["slots"], "slot_sz": s["slot_sz"]}
    if kind == "ref":
        args = (s["probs"], case["smin"], case["smax"], s["states"], s["slots"], s["ctrs"],
                s["acc"])
        s["acc"].zero_()
        for t in range(case["ntries"]):
            H.phase_ref_step(case["n"], case["nallocs"], t, case["niters"], *args)
        H.phase_ref_step(case["n"], case["nallocs"], case["ntries"], case["niters"], *args,
                         rest=True)
        return {"acc": s["acc"], "states": s["states"], "slots": s["slots"], "ctrs": s["ctrs"]}
    if kind == "batched":
        r = s["runner"]
        r.launch(s["handle"])
        return r.d_acc  # (the pointers are all freed again: as many zeros as requests)
    r = H.serve_run(s["results"], case["n"], 1e8, seed=s["seed"])
    return {"results": s["results"], "jobs": r["jobs_done"], "failures": r["alloc_failures"]}


def work(case):
    """Inputs read and outputs written once, the blocks' payload written and
    read back once, and the bit-array words of each malloc/free pair."""
    kind = case["kind"]
    if kind == "grid":
        return {"bytes": case["n"] * (12 + 2 * 16 + META) + case["ncells"] ** 3 * 20, "flops": 0}
    if kind == "strings":
        mean = (case["lo"] + case["hi"]) / 2 + 1
        return {"bytes": case["n"] * (12 + 3 * 8 + 8 * mean + 3 * META), "flops": 0}
    if kind == "graph":
        # the final arrays alone: what a build that knew the degrees would hold
        n, e = case["n"], case["n"] * case["degree"]
        return {"bytes": n * (8 + 4 + 8 + META) + 3 * 4 * e, "flops": 0}
    if kind == "loop":
        pairs = case["n"] * case["nallocs"] * case["niters"]
        return {"bytes": pairs * (2 * 16 + META) + 4 * case["n"], "flops": 0}
    if kind == "phase":
        pairs = case["n"] * case["nslots"] * 0.95 * case["periods"]
        mean = sum(PHASE_SIZES) / len(PHASE_SIZES)
        return {"bytes": pairs * (2 * mean + META + 2 * 12), "flops": 0}
    if kind == "ref":
        # about half of the threads allocate in each step of the schedule
        pairs = 0.5 * 0.91 * case["n"] * case["nallocs"] * case["niters"] * case["ntries"]
        return {"bytes": pairs * (2 * 8 + META) + 16 * case["n"], "flops": 0}
    if kind == "batched":
        hi, lo = case["max_batch"], 1024
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        return {"bytes": case["nbatch"] * mean * (4 + 4 + 2 * 8 + 2 * 8 + META), "flops": 0}
    # mean blocks of a job as the loop draws them (length and lifetime bound it)
    return {"bytes": case["n"] * (180 * (2 * 16 + META) + 16), "flops": 0}
