"""Counts of packed networks around the end of the floats' exact range: an event that takes a
count across it, by any change that a packed network may have, keeps every molecule."""
import numpy as np
import pytest

import oracle
from inchman_b200 import _lib
from inchman_b200.model import DiffusionModel

pytestmark = pytest.mark.gpu

TOP = 1 << 24


def _model(change, nreac, W=16, max_time=0.05):
    m = DiffusionModel(width=W, height=W, physical_length=float(W), p0=0.1, max_time=max_time, output_interval=max_time,
                       solver=_lib.STOCHASTIC_HOMOGENEOUS)
    m.add_species("A", 1.0, 0.0).add_species("B", 0.5, 0.0)
    m.add_reaction("grow", {"A": 1}, {"A": 1, "B": change}, 2e-7)
    m.add_reaction("double", {"A": 1}, {"A": 3}, 2e-7)
    m.add_reaction("own", {"B": 1}, {"B": min(256, change + 1)}, 1e-7)
    for k in range(nreac - 3):
        m.add_reaction(f"rare{k}", {"A": 1}, {"B": 1}, 1e-9)
    return m


def _state(m, change, R, cells):
    """In a few cells, counts that one or two events take to the limit, past it, or that lie beyond."""
    st = np.random.default_rng(change).integers(0, 100, size=(R, 2, m.height, m.width)).astype(np.int32)
    starts = [TOP - k for k in (1, 2, 3, change, change + 1, 2 * change - 1, 255, 256, 257, 513, 0, -3)]
    for r in range(R):
        for i in range(cells):
            st[r, 0, i // m.width, i % m.width] = starts[i % 12]
            st[r, 1, i // m.width, i % m.width] = starts[(i // 12 + 5 * i) % 12]
    return st


@pytest.mark.parametrize("nreac", [3, 9])       # sums in registers, sums in shared memory
@pytest.mark.parametrize("change", [1, 2, 3, 255, 256])
def test_windows_across_the_limit(gpgmp, change, nreac):
    from inchman_b200.solver import Solver
    m = _model(change, nreac)
    desc, keep = m.to_desc()
    R, seed = 2, 50 + change
    st = _state(m, change, R, 250)
    for step in range(3):
        with Solver(m, realisations=R, seed=seed) as s:
            s.set_state(st)
            s.do_reactions(0.5, 640 + step)
            got = s.get_state()
        want = st.copy()
        status = np.zeros(R, np.int32)
        oracle.orc().orc_rep_ssa(oracle.model_ptr(desc), oracle.ptr(want), R, seed, 640 + step, 0.5,
                                 oracle.ptr(status))
        assert np.array_equal(got, want) and not status.any()


@pytest.mark.parametrize("change", [2, 256])
def test_ensembles_across_the_limit(gpgmp, change):
    from inchman_b200.ensemble import Ensemble, InstanceSpec
    import torch
    m = _model(change, 9)
    for r in m.reactions:
        r.rate *= 100.0      # a window is a sixtieth of a second here
    ens = Ensemble([InstanceSpec(m, [0.0, 0.0], 70 + i, 0) for i in range(2)])
    st = _state(m, change, 2, 24)
    state = ens.alloc_state()
    for i in range(2):
        ens.instance_state(state, i).copy_(torch.from_numpy(st[i]))
    ens.run(state)
    ens.results()
    for i in range(2):
        desc, keep = m.to_desc()
        want, _, _, _, _ = oracle.rep_solve(desc, st[i:i + 1], 1, 70 + i, 4)
        assert np.array_equal(ens.instance_state(state, i).cpu().numpy(), want[0])
