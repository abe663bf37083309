"""Strings that do not come from hamalloc: ha_strings_check_c takes them at any
address, ha_strings_concat_c on any 8-byte boundary.  Strings of every length
up to 40 at every offset of a 16-byte granule, one after the other without a
gap, so that what follows a string is the next one's first byte."""
import numpy as np
import pytest

from tests.helpers import allocator

pytestmark = pytest.mark.gpu


def _strings(starts, lengths, gap):
    """One buffer with a string of lengths[i] spaces at starts[i], `gap`
    elsewhere."""
    buf = np.full(int((starts + lengths).max()) + 1, gap, np.uint8)
    for s, n in zip(starts, lengths):
        buf[s:s + n] = ord(" ")
        buf[s + n] = 0
    return buf


@pytest.mark.parametrize("gap", [ord(" "), 0, 255])
def test_check_at_every_offset(torch_cuda, gap):
    import halloc_b200 as H
    torch = torch_cuda
    lengths = np.tile(np.arange(41), 16)
    starts = np.zeros(len(lengths), np.int64)
    at = 0
    for i in range(len(lengths)):
        at += (i // 41 - at) % 16  # offset i // 41 of a granule
        starts[i] = at
        at += int(lengths[i]) + 1
    buf = torch.from_numpy(_strings(starts, lengths, gap)).cuda()
    assert buf.data_ptr() % 16 == 0
    n = len(lengths)
    ptrs = torch.from_numpy(starts + buf.data_ptr()).cuda()
    zero = torch.zeros(n, dtype=torch.int32, device="cuda")
    bad = torch.zeros(3, dtype=torch.int64, device="cuda")
    with allocator(memory=256 << 20):
        for k, off in enumerate((0, 1, -1)):
            # the wanted length given in the first or in the second array
            want = torch.from_numpy((lengths + off).clip(0).astype(np.int32)).cuda()
            args = (want, zero) if k != 1 else (zero, want)
            H.strings_check(n, ptrs, *args, bad[k:])
        torch.cuda.synchronize()
    assert bad.tolist() == [0, n, n - int((lengths == 0).sum())]


def test_concat_on_word_boundaries(torch_cuda):
    import halloc_b200 as H
    torch = torch_cuda
    rng = np.random.default_rng(7)
    n = 2000
    bufs, ptrs, lens = [], [], []
    for _ in range(2):
        lengths = rng.integers(0, 41, n)
        starts = np.cumsum(np.concatenate([[8], lengths[:-1] // 8 * 8 + 8 + 8 * rng.integers(0, 2, n - 1)]))
        buf = torch.from_numpy(_strings(starts, lengths, 255)).cuda()
        bufs.append(buf)
        ptrs.append(torch.from_numpy(starts + buf.data_ptr()).cuda())
        lens.append(torch.from_numpy(lengths.astype(np.int32)).cuda())
    with allocator(memory=256 << 20):
        c = torch.zeros(n, dtype=torch.int64, device="cuda")
        cnt = torch.zeros(2, dtype=torch.int64, device="cuda")
        H.strings_concat(n, c, ptrs[0], ptrs[1], cnt)
        H.strings_check(n, c, lens[0], lens[1], cnt[1:])
        H.strings_free(n, c)
        torch.cuda.synchronize()
        assert cnt.tolist() == [0, 0]
        st = H.stats()
        assert st["used_chunks"] == 0 and st["status"] == 0
