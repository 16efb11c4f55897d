"""Gray-Scott solves whose outputs lie on their inputs: in place, with the fields exchanged, in
overlapping parts of one buffer, and with the first checkpoint as the initial state."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forward(dtype, p, u0, v0, u, v, ck=None):
    import torch
    from inchman_b200 import _lib
    from inchman_b200 import gray_scott as gs
    name = "gpgmp_gs_forward_f64" if dtype == np.float64 else "gpgmp_gs_forward_f32"
    args = [C.c_void_p(t.data_ptr()) if t is not None else None for t in (u0, v0, u, v, ck)]
    _lib.check(gs._fn(name)(C.byref(p), *args, C.c_void_p(torch.cuda.current_stream().cuda_stream)), name)


@pytest.mark.parametrize("dtype,n", [(np.float32, 33), (np.float32, 100), (np.float32, 192), (np.float32, 320),
                                     (np.float64, 96), (np.float64, 256)])
@pytest.mark.parametrize("steps", [0, 1, 7, 8, 9, 25])
def test_outputs_on_inputs(gpgmp, dtype, n, steps):
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=n, steps=steps, vx=0.05, vy=-0.03)
    a, b = (torch.from_numpy(x).cuda() for x in cfg.initial_state(dtype))
    p = cfg.params(checkpoint_every=3)
    want = gs.forward(a, b, p)
    # float64: the cluster kernel's rounding, carried on with a factor below 1.2 a step
    tol = 0.0 if dtype == np.float32 else 8 * 2.0 ** -52 * sum(1.2 ** k for k in range(steps))

    def check(u, v):
        torch.cuda.synchronize()
        assert gs.status() == 0
        for x, y in zip((u, v), want):
            assert float((x - y).abs().max()) <= tol

    u, v = a.clone(), b.clone()
    _forward(dtype, p, u, v, u, v)
    check(u, v)
    u, v = a.clone(), b.clone()
    _forward(dtype, p, u, v, v, u)
    check(v, u)
    buf = torch.cat([a.flatten(), b.flatten(), a.flatten()])
    u0, v0, u = buf[:n * n], buf[n * n:2 * n * n], buf[5 * n + 3:n * n + 5 * n + 3]
    v = torch.empty_like(b)
    _forward(dtype, p, u0, v0, u, v)
    check(u.view(n, n), v)
    ck = torch.zeros((max(1, -(-steps // 3)), 2, n, n), dtype=a.dtype, device="cuda")
    ck[0, 0], ck[0, 1] = a, b
    u, v = torch.empty_like(a), torch.empty_like(b)
    _forward(dtype, p, ck[0, 0], ck[0, 1], u, v, ck)
    check(u, v)
    assert torch.equal(ck[0, 0], a) and torch.equal(ck[0, 1], b)


@pytest.mark.parametrize("variant,steps", [(0, 1), (0, 8), (0, 9), (0, 40), (42, 16), (42, 17), (40, 3)])
def test_several_clusters(gpgmp, variant, steps):
    """The multi-cluster families at n = 256 (8 or 16 ghost rows)."""
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=256, steps=steps)
    a, b = (torch.from_numpy(x).cuda() for x in cfg.initial_state(np.float32))
    p = cfg.params(variant=variant)
    want = gs.forward(a, b, p)
    u, v = a.clone(), b.clone()
    _forward(np.float32, p, u, v, u, v)
    assert gs.status() == 0 and torch.equal(u, want[0]) and torch.equal(v, want[1])
    buf = torch.cat([a.flatten(), b.flatten(), a.flatten()])
    u0, v0, u = buf[:65536], buf[65536:131072], buf[65536 + 4096:131072 + 4096]
    v = torch.empty_like(b)
    _forward(np.float32, p, u0, v0, u, v)
    assert gs.status() == 0 and torch.equal(u.view(256, 256), want[0]) and torch.equal(v, want[1])
