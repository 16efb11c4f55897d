"""The tiled Gray-Scott kernel (variant 50) against the kernels it stands in for: float32 bit
for bit at step counts around its swap period, for sides with one tile, a ragged last tile,
odd sides and both arithmetics; float64 to a few roundings per step; the register-resident
float64 kernels against the column walk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(n, steps, drift, dtype, variant, every=0):
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=n, steps=steps, vx=0.05 if drift else 0.0, vy=-0.03 if drift else 0.0)
    u0, v0 = (torch.from_numpy(a).cuda() for a in cfg.initial_state(dtype))
    ck = None
    if every:
        ck = torch.zeros((-(-steps // every), 2, n, n), dtype=u0.dtype, device="cuda")
    u, v = gs.forward(u0, v0, cfg.params(variant=variant, checkpoint_every=every or 100), checkpoints=ck)
    assert gs.status() == 0
    return [u, v] + ([ck] if every else [])


@pytest.mark.parametrize("n,steps,drift,every,ref", [
    (24, 9, True, 0, 1), (33, 17, False, 3, 1), (48, 8, True, 1, 1), (75, 25, True, 4, 1), (96, 7, False, 2, 1),
    (100, 33, False, 5, 1), (160, 16, True, 0, 1), (192, 41, True, 10, 1), (320, 24, False, 0, 1),
    (64, 33, True, 7, 3), (128, 17, False, 1, 3), (256, 34, True, 8, 3), (96, 0, False, 0, 1), (256, 1, False, 1, 3)])
def test_float32_tiles_give_the_same_bits(gpgmp, n, steps, drift, every, ref):
    import torch
    a, b = _run(n, steps, drift, np.float32, 50, every), _run(n, steps, drift, np.float32, ref, every)
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("n,steps,drift,variant", [(96, 33, True, 50), (75, 17, False, 50), (256, 25, True, 50),
                                                   (64, 41, True, 0), (64, 8, False, 0), (128, 33, False, 0),
                                                   (128, 17, True, 0)])
def test_float64_kernels_agree(gpgmp, n, steps, drift, variant):
    # a step's rounding (2^-52 of values below 2) is carried on with a factor below 1.2 a step
    a, b = _run(n, steps, drift, np.float64, variant, 4), _run(n, steps, drift, np.float64, 1, 4)
    tol = 8 * 2.0 ** -52 * sum(1.2 ** k for k in range(steps))
    for x, y in zip(a, b):
        assert float((x - y).abs().max()) <= tol


def test_tiles_on_two_streams(gpgmp):
    """Two solves at once have their own exchange buffers and wait for room on the chip."""
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=320, steps=80)
    u0, v0 = (torch.from_numpy(a).cuda() for a in cfg.initial_state(np.float32))
    ref = gs.forward(u0, v0, cfg.params())
    torch.cuda.synchronize()
    got = []
    for s in [torch.cuda.Stream() for _ in range(4)]:
        with torch.cuda.stream(s):
            got.append(gs.forward(u0, v0, cfg.params()))
    torch.cuda.synchronize()
    for u, v in got:
        assert torch.equal(u, ref[0]) and torch.equal(v, ref[1])
    assert gs.status() == 0
