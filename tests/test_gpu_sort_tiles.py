"""Radix sort of long lists at the edges of the tiles (9216 keys for 8-bit digits, 7680 for
10-bit ones) and of the digit counts' 16-byte loads, against the oracle's stable sort."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 13, 20, 24, 30, 32])
@pytest.mark.parametrize("n", [8193, 9215, 9216, 9217, 15360, 15361, 18432, 55299, 300007])
@pytest.mark.parametrize("spread", ["uniform", "few", "top"])
def test_long_sorts(gpgmp, n, bits, spread):
    import torch
    from inchman_b200 import individual as ind
    rng = np.random.default_rng(n * 41 + bits)
    hi = (1 << bits) - 1
    keys = rng.integers(0, hi + 1, size=n, dtype=np.uint64).astype(np.uint32)
    if spread == "few":
        keys %= 5
    elif spread == "top":
        keys[:] = hi
    vals = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    wk, wv = keys.copy(), vals.copy()
    oracle.orc().orc_sort_pairs_u32(oracle.ptr(wk), oracle.ptr(wv), n)
    off = n % 4                      # lists that start on any 4-byte boundary
    k = torch.zeros(n + off, dtype=torch.int32, device="cuda")[off:]
    k.copy_(torch.from_numpy(keys.view(np.int32)))
    ko, vo, scratch = ind.sort_pairs_u32(k, torch.from_numpy(vals.view(np.int32)).cuda(), bits)
    assert np.array_equal(ko.cpu().numpy().view(np.uint32), wk)
    assert np.array_equal(vo.cpu().numpy().view(np.uint32), wv)
    assert ind.scratch_status(scratch, 1, n, bits) == 0


def test_equal_keys_past_a_16_bit_counter(gpgmp):
    """So many equal keys that a lane's counter of the 10-bit digits would wrap."""
    import torch
    from inchman_b200 import individual as ind
    n, bits = 148 * 96 * 16384 + 70001, 20
    k = torch.full((n,), 0x5A5A5, dtype=torch.int32, device="cuda")
    k[n // 3] = 7
    k[n // 2] = 0xFFFFF
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo, scratch = ind.sort_pairs_u32(k, v, bits)
    assert ind.scratch_status(scratch, 1, n, bits) == 0
    assert ko[0] == 7 and ko[-1] == 0xFFFFF and bool((ko[1:-1] == 0x5A5A5).all())
    keep = torch.cat([v[:n // 3], v[n // 3 + 1:n // 2], v[n // 2 + 1:]])
    assert vo[0] == n // 3 and vo[-1] == n // 2 and torch.equal(vo[1:-1], keep)
