"""The tiled adjoint (sides without a kernel of their own) against the cluster kernel that runs
under variant 1: lattices of one tile, ragged and odd ones, segments around the swap period."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,steps,every,drift", [(24, 9, 4, True), (33, 17, 17, False), (75, 25, 8, True),
                                                 (96, 33, 16, False), (100, 7, 1, True), (192, 41, 9, True),
                                                 (160, 16, 16, False)])
def test_tiled_adjoint(gpgmp, n, steps, every, drift, dtype):
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=n, steps=steps, vx=0.05 if drift else 0.0, vy=-0.03 if drift else 0.0)
    u0, v0 = (torch.from_numpy(a).cuda() for a in cfg.initial_state(dtype))
    g = torch.Generator(device="cuda").manual_seed(n)
    up = [torch.randn((n, n), generator=g, device="cuda", dtype=u0.dtype) for _ in range(2)]
    out = {}
    for variant in (0, 1):
        p = cfg.params(variant=variant, checkpoint_every=every)
        ck = torch.zeros((-(-steps // every), 2, n, n), dtype=u0.dtype, device="cuda")
        gs.forward(u0, v0, p, checkpoints=ck)
        out[variant] = gs.adjoint(p, ck, *up)
    assert gs.status() == 0
    # float32: the same operations; float64: a rounding per step carried on with a factor
    # below 1.2, of values below 8
    tol = 0.0 if dtype == np.float32 else 64 * 2.0 ** -52 * sum(1.2 ** k for k in range(steps))
    for x, y in zip(out[0][:2], out[1][:2]):
        assert float((x - y).abs().max()) <= tol
    # the sums are in double on both sides: their order, and for float64 the fields' rounding
    scale = steps * n * n
    assert float((out[0][2] - out[1][2]).abs().max()) <= max(scale * 2.0 ** -52 * 64, tol * scale)
