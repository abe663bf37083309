"""Builds tests/hostcore/hostcore.cpp against the core's present source and
binds it."""
import ctypes
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
CSRC = os.path.join(ROOT, "halloc_b200", "csrc")
INCLUDE = os.path.join(ROOT, "include")
NSIZES, NHEADS, NONE = 16, 16, 0xFFFFFFFF


def build(out_dir, csrc=CSRC, include=INCLUDE):
    so = os.path.join(str(out_dir), "hostcore.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-w", "-U_FORTIFY_SOURCE",
                    "-I" + HERE, "-I" + csrc, "-I" + include,
                    os.path.join(HERE, "hostcore.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _odd_prime_below(n, nb):
    for p in range(n - 1, 2, -1):
        if all(p % d for d in range(2, int(p ** 0.5) + 1)) and n % p and nb % p:
            return p
    return 3


def classes(sb_bytes, busy=0.835, roomy=0.6, sparse=0.012):
    """The size table (nchunks, chunk_enc, chunk_id, ncib, sparse, hash_step,
    roomy, busy) of slabs of sb_bytes, as halloc.cu builds it; a hash step
    where the rule has none is 3 blocks."""
    t = np.zeros((NSIZES, 8), np.uint32)
    for sid in range(NSIZES):
        unit = 8 << (sid // 2)
        block = (3 if sid & 1 else 2) * unit
        slot = 4 if sid < 2 else 2 if sid < 4 else 1
        nblocks = sb_bytes // block // slot * slot
        cid = (sid & 1) + (0 if sid < NSIZES // 2 else 2)
        cbytes = (3 if cid & 1 else 2) * (128 if cid >= 2 else 8)
        ncib = block // cbytes
        n = nblocks * ncib
        three = cbytes % 3 == 0
        enc = (3 if three else 1) << 16 | (cbytes // 3 if three else cbytes).bit_length() - 1
        span = min(max(nblocks // 256 + nblocks // 64, 4), nblocks)
        t[sid] = [n, enc, cid, ncib, int(sparse * n), ncib * _odd_prime_below(span, nblocks),
                  int(roomy * n), int(busy * n)]
    return t


class Core:
    def __init__(self, lib):
        self.lib = lib
        lib.hc_run.restype = ctypes.c_int64

    def init(self, nsbs, sb_sh=16, nheads=1, surge=1, **fractions):
        self.nsbs, self.sb_sh = nsbs, sb_sh
        self.cls = classes(1 << sb_sh, **fractions)
        # one-chunk sizes count early, as in the library
        spec = sum(1 << s for s in range(NSIZES) if self.cls[s, 3] == 1)
        self.lib.hc_init(nsbs, sb_sh, self.cls.ctypes.data_as(ctypes.c_void_p), nheads, surge, spec)

    def run(self, programs, seed, sm=None, hold=200, max_points=20_000_000):
        """programs: per warp an int array (ops, lanes): size > 0 allocates, -k - 1
        frees the lane's result of op k.  Returns the results (offset, -1 NULL,
        -2 freed) in the same shapes."""
        progs = [np.ascontiguousarray(p, np.int64).reshape(len(p), -1) for p in programs]
        res = [np.full(p.shape, -3, np.int64) for p in progs]
        n = len(progs)
        pp = (ctypes.c_void_p * n)(*[p.ctypes.data for p in progs])
        rr = (ctypes.c_void_p * n)(*[r.ctypes.data for r in res])
        lanes = np.array([p.shape[1] for p in progs], np.uint32)
        nops = np.array([len(p) for p in progs], np.int64)
        sm = np.array(range(n) if sm is None else sm, np.uint32)
        pts = self.lib.hc_run(n, lanes.ctypes.data_as(ctypes.c_void_p),
                              sm.ctypes.data_as(ctypes.c_void_p), pp,
                              nops.ctypes.data_as(ctypes.c_void_p), rr, ctypes.c_uint64(seed),
                              hold, ctypes.c_int64(max_points))
        assert pts >= 0, "the warps came to no end"
        return res

    def head(self, sid, k=0):
        out = (ctypes.c_uint32 * 4)()
        self.lib.hc_head(sid, k, out)
        return dict(zip(("slab", "prefetched", "level", "level_copy"), out))

    def slab(self, sb):
        out = (ctypes.c_uint32 * 7)()
        self.lib.hc_slab(sb, out)
        return dict(zip(("used", "head_flag", "chunk", "size_id", "chunk_id", "is_head", "nsets"),
                        out))

    status = property(lambda self: self.lib.hc_status())
    nulls = property(lambda self: self.lib.hc_nulls())
    head_changes = property(lambda self: self.lib.hc_head_changes())
    surge_changes = property(lambda self: self.lib.hc_surge_changes())
    level_moves = property(lambda self: self.lib.hc_level_moves())
