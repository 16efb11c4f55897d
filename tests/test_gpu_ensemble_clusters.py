"""Ensembles whose instances are shared by a cluster of CTAs (few instances, or one that
outlasts the rest): every instance keeps the bits of its own solver, with snapshots, absorbing
walls, areas that are no multiple of a warp, networks that do not fit the packed form and
counts beyond the floats' exact range."""
import numpy as np
import pytest

from helpers import small_homog

pytestmark = pytest.mark.gpu


def _big_stoich(m):
    m.add_reaction("burst", {"A": 1}, {"C": 300}, 0.02)      # a change of 300: not packed
    return m


@pytest.mark.parametrize("sizes,threads,kind", [
    ([32], 1024, ""), ([45, 17, 33], 1024, ""), ([64] * 16, 1024, ""), ([20] * 40, 256, ""), ([96] + [16] * 20, 512, ""),
    ([33, 21], 1024, "unpacked"), ([24], 1024, "large")])
def test_instances_match_their_solvers(gpgmp, sizes, threads, kind):
    import torch
    from inchman_b200.ensemble import Ensemble, InstanceSpec
    from inchman_b200.solver import Solver
    specs = []
    for i, w in enumerate(sizes):
        m = small_homog(W=w, H=w, max_time=0.12, bmask=(0, i % 2, 0, 1))
        m.output_interval = 0.05
        if kind == "unpacked":
            _big_stoich(m)
        specs.append(InstanceSpec(m, [60.0, 40.0, 5.0], 100 + i, 0, max_snapshots=5))
    ens = Ensemble(specs)
    ens.configure(threads, 1)
    state, snaps = ens.alloc_state(), ens.alloc_snapshots()
    ens.init_poisson(state)
    if kind == "large":      # a cell that starts beyond 2^24, and one that grows past it
        s0 = ens.instance_state(state, 0)
        s0[0, 3, 4] = (1 << 24) + 5
        s0[0, 10, 10] = (1 << 24) - 3
        s0[1, 10, 10] = 0
        s0[2, 10, 10] = 60
    init = state.clone()
    ens.run(state, snaps)
    status, steps, times = ens.results()
    for i in sorted({0, len(specs) // 2, len(specs) - 1}):
        sp = specs[i]
        with Solver(sp.model, realisations=1, seed=sp.seed) as s:
            s.set_state(ens.instance_state(init, i).cpu().numpy()[None])
            got, t, n = s.solve(max_snapshots=5)
            assert n == steps[i] and np.array_equal(s.status(), status[i:i + 1])
            assert np.array_equal(s.get_state()[0], ens.instance_state(state, i).cpu().numpy())
        o, block = ens.snap_offsets[i], int(np.prod(ens.shapes[i]))
        mine = snaps[o:o + len(got) * block].cpu().numpy().reshape(got[:, 0].shape)
        assert np.array_equal(mine, got[:, 0])
        assert np.array_equal(times[5 * i:5 * i + len(t)], t)
    assert torch.cuda.is_available()
