"""Calls captured into a CUDA graph and replayed on new inputs: the tiled Gray-Scott forward and
adjoint, a batch, and the list primitives in their short and long forms."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _capture(fn):
    """Warm up on a side stream, capture, and return the graph."""
    import torch
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        fn()
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fn()
    return g


@pytest.mark.parametrize("dtype,n,steps", [(np.float32, 96, 40), (np.float32, 33, 17), (np.float64, 96, 25),
                                           (np.float64, 128, 30), (np.float64, 256, 17), (np.float32, 256, 24)])
def test_gray_scott(gpgmp, dtype, n, steps):
    import torch
    from inchman_b200 import _lib
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=n, steps=steps)
    p = cfg.params(checkpoint_every=10)
    kind = "f64" if dtype == np.float64 else "f32"
    eb = np.dtype(dtype).itemsize
    ckb, wb = gs.buffer_sizes(p, eb)
    a, b = (torch.from_numpy(x).cuda() for x in cfg.initial_state(dtype))
    u, v, gu, gv = (torch.zeros_like(a) for _ in range(4))
    ck = torch.zeros(ckb // eb, dtype=a.dtype, device="cuda")
    work = torch.zeros(wb // eb, dtype=a.dtype, device="cuda")
    g6 = torch.zeros(6, dtype=torch.float64, device="cuda")

    def call(name, *ts):
        name = f"gpgmp_gs_{name}_{kind}"
        _lib.check(gs._fn(name)(C.byref(p), *[C.c_void_p(t.data_ptr()) for t in ts],
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)), name)

    def run():
        call("forward", a, b, u, v, ck)
        call("adjoint", ck, u, v, gu, gv, g6, work)
    graph = _capture(run)
    for k in range(3):
        a.add_(0.01)
        graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (u, v, gu, gv)]
        run()
        torch.cuda.synchronize()
        assert gs.status() == 0
        for x, y in zip(got, (u, v, gu, gv)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("n", [700, 5000, 20000, 200 * 16384 + 3])
def test_lists(gpgmp, n):
    import torch
    from inchman_b200 import individual as ind
    bits, ncells = 10, 1000
    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, ncells, (n,), generator=g, device="cuda", dtype=torch.int32)
    vals = torch.arange(n, device="cuda", dtype=torch.int32)
    ko, vo, sc = torch.empty_like(keys), torch.empty_like(vals), torch.empty_like(keys)
    start, count = (torch.empty(ncells, device="cuda", dtype=torch.int32) for _ in range(2))
    ss, ws, cs = ind.sort_scratch(n, bits), ind.scan_scratch(n), ind.scan_scratch(ncells)
    p = ind._ptr

    def run():
        ind._call("gpgmp_sort_pairs_u32", p(keys), p(vals), p(ko), p(vo), n, bits, p(ss), ss.numel(), ind._stream())
        ind._call("gpgmp_cell_offsets", p(ko), n, ncells, p(start), p(count), p(cs), cs.numel(), ind._stream())
        ind._call("gpgmp_exclusive_scan_u32", p(keys), p(sc), n, p(ws), ws.numel(), ind._stream())
    graph = _capture(run)
    for k in range(3):
        keys.copy_(torch.randint(0, ncells, (n,), generator=g, device="cuda", dtype=torch.int32))
        graph.replay()
        torch.cuda.synchronize()
        order = torch.sort(keys, stable=True)
        assert torch.equal(ko, order.values) and torch.equal(vo.long(), order.indices)
        c = torch.bincount(keys.long(), minlength=ncells)
        assert torch.equal(count.long(), c) and torch.equal(start.long(), torch.cumsum(c, 0) - c)
        x = keys.long()
        assert torch.equal(sc.long() & 0xFFFFFFFF, (torch.cumsum(x, 0) - x) & 0xFFFFFFFF)


@pytest.mark.parametrize("batch", [1, 20, 96, 97, 200])
def test_batch(gpgmp, batch):
    """The members' parameters are part of the captured call."""
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=64, steps=30)
    a, b = (torch.from_numpy(x).cuda() for x in cfg.initial_state(np.float32))
    u0, v0 = a.repeat(batch, 1, 1), b.repeat(batch, 1, 1)
    mp = np.tile(np.array(cfg.theta()), (batch, 1))
    mp[:, 0] += np.arange(batch) * 1e-4
    out = {}

    def run():
        out["u"], out["v"] = gs.forward_batch(u0, v0, cfg.params(), mp.copy())
    graph = _capture(run)
    for k in range(2):
        u0.add_(torch.linspace(0, 0.02, batch, device="cuda").view(batch, 1, 1))
        graph.replay()
        torch.cuda.synchronize()
        for m in {0, batch // 2, batch - 1}:
            u, v = gs.forward(u0[m].clone(), v0[m].clone(), cfg.params(F=mp[m, 0]))
            assert torch.equal(u, out["u"][m]) and torch.equal(v, out["v"][m])
