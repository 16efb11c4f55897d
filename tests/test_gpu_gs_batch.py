"""Batched Gray-Scott forward: every kernel that a batch can take (16-CTA clusters and row
blocks on 8, 4, 2 and 1 CTAs) gives each member the bits of its own single solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# lattice side, batch (one on each side of the choices' borders), steps, drift
@pytest.mark.parametrize("n,batch,steps,drift", [
    (64, 8, 7, False), (64, 30, 8, True), (64, 70, 1, False), (64, 96, 9, True), (64, 260, 6, False),
    (128, 8, 5, True), (128, 12, 8, False), (128, 60, 9, True), (128, 90, 4, False), (128, 90, 7, True),
    (256, 6, 3, False), (256, 12, 6, True), (256, 20, 5, False), (256, 20, 1, True), (64, 70, 0, False),
])
def test_batch_members_are_their_single_solves(gpgmp, n, batch, steps, drift):
    import torch
    from inchman_b200 import gray_scott as gs
    cfg = gs.GrayScottConfig(n=n, steps=steps, vx=0.04 if drift else 0.0, vy=-0.02 if drift else 0.0)
    u0, v0 = (torch.from_numpy(a).cuda() for a in cfg.initial_state())
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    u = u0 + 0.01 * torch.rand((batch, n, n), generator=g, device="cuda")
    v = v0 + 0.01 * torch.rand((batch, n, n), generator=g, device="cuda")
    th = np.tile(cfg.theta(), (batch, 1))
    th[:, 0] *= np.linspace(0.9, 1.1, batch)
    bu, bv = gs.forward_batch(u, v, cfg.params(), member_params=th)
    for m in (0, 1, batch // 2, batch - 1):
        su, sv = gs.forward(u[m], v[m], cfg.params(F=th[m, 0]))
        assert torch.equal(bu[m], su) and torch.equal(bv[m], sv), m
    assert gs.status() == 0
