"""Exclusive scan over more tiles than SMs (the streaming kernel): whole rounds, one tile more
or less, a partial last tile, a stage's reuse of its buffer, in place, and an unaligned view
of the same size (the look-back kernel)."""
import pytest

pytestmark = pytest.mark.gpu

TILE = 16384


@pytest.mark.parametrize("rounds,tiles,extra", [(1, 1, 0), (1, 1, 5), (2, -1, 0), (2, 0, 0), (3, 0, -1), (3, 1, 1),
                                                (4, 17, 8191), (5, 0, 4)])
def test_streaming_scan(gpgmp, rounds, tiles, extra):
    import torch
    from inchman_b200 import individual as ind
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (rounds * sms + tiles) * TILE + extra
    g = torch.Generator(device="cuda").manual_seed(n)
    whole = torch.randint(-(1 << 31), 1 << 31, (n + 1,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    for x in (whole[:n], whole[1:]):
        want = (torch.cumsum(x.to(torch.int64) & 0xFFFFFFFF, 0) - (x.to(torch.int64) & 0xFFFFFFFF)) & 0xFFFFFFFF
        scratch = ind.scan_scratch(n)
        got = ind.exclusive_scan_u32(x, scratch)
        assert ind.scratch_status(scratch, 0) == 0
        assert torch.equal(got.to(torch.int64) & 0xFFFFFFFF, want)
    x = whole[:n].clone()
    want = (torch.cumsum(x.to(torch.int64) & 0xFFFFFFFF, 0) - (x.to(torch.int64) & 0xFFFFFFFF)) & 0xFFFFFFFF
    scratch = ind.scan_scratch(n)
    ind._call("gpgmp_exclusive_scan_u32", ind._ptr(x), ind._ptr(x), n, ind._ptr(scratch), scratch.numel(), ind._stream())
    assert torch.equal(x.to(torch.int64) & 0xFFFFFFFF, want)
