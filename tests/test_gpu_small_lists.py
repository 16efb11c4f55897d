"""One-launch sorts and cell offsets of short lists, at the edges of their item counts and
ranges: against the oracle's stable sort, and a histogram and its sums."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _np(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n,bits", [(1, 1), (2, 32), (31, 5), (33, 6), (1023, 10), (1024, 32), (1025, 7), (2048, 4),
                                    (2049, 31), (4095, 20), (4096, 9), (4097, 11), (8191, 32), (8192, 13), (8193, 13)])
@pytest.mark.parametrize("spread", ["uniform", "few", "top"])
def test_short_sorts(gpgmp, n, bits, spread):
    from inchman_b200 import individual as ind
    rng = np.random.default_rng(n * 37 + bits)
    hi = (1 << bits) - 1
    keys = rng.integers(0, hi + 1, size=n, dtype=np.uint64).astype(np.uint32)
    if spread == "few":
        keys %= 3
    elif spread == "top":
        keys[:] = hi            # every digit at its largest value, as the padding's
    vals = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    wk, wv = keys.copy(), vals.copy()
    oracle.orc().orc_sort_pairs_u32(oracle.ptr(wk), oracle.ptr(wv), n)
    ko, vo, scratch = ind.sort_pairs_u32(_t(keys), _t(vals), bits)
    assert np.array_equal(_np(ko), wk) and np.array_equal(_np(vo), wv)
    assert ind.scratch_status(scratch, 1, n, bits) == 0


def test_short_sort_by_low_bits_only(gpgmp):
    """Bits above key_bits are carried, not compared."""
    from inchman_b200 import individual as ind
    rng = np.random.default_rng(4)
    keys = rng.integers(0, 1 << 32, size=3000, dtype=np.uint64).astype(np.uint32)
    order = np.argsort(keys & 0x7F, kind="stable")
    ko, vo, _ = ind.sort_pairs_u32(_t(keys), _t(np.arange(3000, dtype=np.uint32)), 7)
    assert np.array_equal(_np(ko), keys[order]) and np.array_equal(_np(vo), order.astype(np.uint32))


@pytest.mark.parametrize("n,cells", [(0, 1), (1, 1), (5, 3), (1000, 1023), (4096, 1024), (4097, 1025), (32768, 16384),
                                     (32769, 16384), (32768, 16385), (777, 16383)])
def test_cell_offsets_of_short_lists(gpgmp, n, cells):
    from inchman_b200 import individual as ind
    rng = np.random.default_rng(n + cells)
    keys = np.sort(rng.integers(0, cells + 3, size=n)).astype(np.uint32)      # some past the last cell
    scratch = ind.scan_scratch(cells)
    start, count = ind.cell_offsets(_t(keys), cells, scratch)
    want = np.bincount(keys, minlength=cells + 3)[:cells].astype(np.uint32)
    assert np.array_equal(_np(count), want)
    assert np.array_equal(_np(start), np.concatenate([[0], np.cumsum(want)[:-1]]).astype(np.uint32))
    assert ind.scratch_status(scratch, 0) == 0
