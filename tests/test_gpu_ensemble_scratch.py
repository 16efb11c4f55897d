"""Device memory of an ensemble whose instances are wide and many (one CTA each): the scratch of the
jumps is one buffer per CTA at work, and the results are those of the instances' own solvers."""
import numpy as np
import pytest

from helpers import small_homog

pytestmark = pytest.mark.gpu


def _specs(n, w, max_time):
    from inchman_b200.ensemble import InstanceSpec
    m = small_homog(W=w, H=w, max_time=max_time, bmask=(0, 1, 0, 0))
    m.output_interval = max_time
    return [InstanceSpec(m, [6.0, 4.0, 1.0], 300 + i, 0) for i in range(n)]


def _bytes(specs):
    import torch
    from inchman_b200.ensemble import Ensemble
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ens = Ensemble(specs)
    used = before - torch.cuda.mem_get_info()[0]
    return ens, used


def test_wide_instances_one_buffer_per_cta(gpgmp):
    import torch
    ctas = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    ens, used = _bytes(_specs(ctas + 8, 512, 0.1))
    t, per_sm, grid = ens.launch_shape()
    one = 16 * 512 * 512
    assert used <= (grid + 8) * one + (64 << 20)


def test_few_instances_no_more_buffers_than_instances(gpgmp):
    ens, used = _bytes(_specs(3, 1024, 0.1))
    assert used <= 2 * 3 * 16 * 1024 * 1024 + (64 << 20)


@pytest.mark.parametrize("w", [128, 132])      # two lost buffers, and one
def test_results(gpgmp, w):
    import torch
    from inchman_b200.ensemble import Ensemble
    from inchman_b200.solver import Solver
    # as many as CTAs fit at once: a cluster each would take two rounds
    per_sm = Ensemble(_specs(1, w, 0.06)).launch_shape()[1]
    specs = _specs(per_sm * torch.cuda.get_device_properties(0).multi_processor_count, w, 0.06)
    ens = Ensemble(specs)
    state = ens.alloc_state()
    ens.init_poisson(state)
    init = state.clone()
    ens.run(state)
    status, steps, _ = ens.results()
    for i in (0, 5, len(specs) - 1):
        with Solver(specs[i].model, realisations=1, seed=specs[i].seed) as s:
            s.set_state(ens.instance_state(init, i).cpu().numpy()[None])
            _, _, n = s.solve(max_snapshots=2)
            assert n == steps[i]
            assert np.array_equal(s.get_state()[0], ens.instance_state(state, i).cpu().numpy())
