"""Drift-diffusion sweeps on grids whose rows need more tiles than a launch has in one dimension."""
import numpy as np
import pytest

import oracle
from helpers import small_inhom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(3, 524281), (2, 1048553), (600011, 2)])
def test_tall_and_wide_grids(gpgmp, W, H):
    from inchman_b200.solver import Solver
    m = small_inhom(W=8, H=8)
    m.width, m.height = W, H
    m.reactions = []
    rng = np.random.default_rng(W)
    D = rng.lognormal(0.0, 0.5, size=(H, W)).astype(np.float32)
    rx, ry = (rng.uniform(-0.3, 0.3, size=(H, W)).astype(np.float32) for _ in range(2))
    m.field_dx = np.stack([D, D]); m.field_dy = np.stack([D, D])
    m.field_rx = np.stack([rx, rx]); m.field_ry = np.stack([ry, ry])
    desc, keep = m.to_desc()
    fields = [np.ascontiguousarray(f, dtype=np.float32) for f in (m.field_dx, m.field_dy, m.field_rx, m.field_ry)]
    st = rng.integers(0, 60, size=(1, 2, H, W)).astype(np.int32)
    seed = 5
    with Solver(m, realisations=1, seed=seed) as s:
        dtx, dty = s.timesteps()
        s.set_state(st)
        s.diffuse(1, float(max(dtx[1], dty[1])), 128)
        got = s.get_state()
    want = st.copy()
    for d, dt in ((0, dtx), (1, dty)):
        oracle.orc().orc_rep_inhomog_sweep(oracle.model_ptr(desc), oracle.ptr(want), 1, seed, 1, d, 128 + d, float(dt[1]),
                                           oracle.ptr(fields[d]), oracle.ptr(fields[2 + d]))
    assert np.array_equal(got, want)
