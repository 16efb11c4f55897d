"""The particle step at each number and width of its sort's digits (grids of 1 cell to
2^30) and at counts around its warps and blocks, against the CPU oracle, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [1, 16, 100, 256, 300, 1024, 2000, 4097])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 20011])
def test_particle_steps(gpgmp, grid, n):
    from inchman_b200 import individual as ind
    steps, D, vx, vy, dt, p_react, seed = 2, 0.5, 0.1, -0.05, 1.0, 0.3, 11
    x, y, sp = ind.uniform_particles(n, grid, seed=3)
    p = ind.Particles(n, grid, D=D, vx=vx, vy=vy, dt=dt, p_react=p_react, seed=seed)
    p.set(x, y, sp)
    p.step(steps)
    gx, gy, gs = p.get()
    ox, oy, osp = x.copy(), y.copy(), sp.copy()
    m = oracle.orc().orc_particles_run(n, oracle.ptr(ox), oracle.ptr(oy), oracle.ptr(osp), grid, D, vx, vy, dt,
                                       p_react, seed, 0, steps)
    assert gx.size == m
    assert np.array_equal(gx.view(np.uint32), ox[:m].view(np.uint32))
    assert np.array_equal(gy.view(np.uint32), oy[:m].view(np.uint32))
    assert np.array_equal(gs, osp[:m])


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 2304, 2305, 6145, 45_000, 44_999, 65_536, 65_537,
                               67_584, 67_840, 67_841, 100_003, 262_149])
@pytest.mark.parametrize("shape", ["uniform", "corners", "one_cell", "end"])
def test_particle_bins_and_pairs(gpgmp, n, shape):
    """Lists around the tiles of the sorted list, and cells of up to all particles with long
    runs of empty cells before, between and after them: positions, and the bins of the step."""
    from inchman_b200 import individual as ind
    grid = 40 if n < 40_000 else 300 if n < 200_000 else 1024
    D, p_react, seed = 0.02, 0.4, 5
    rng = np.random.default_rng(n)
    x = rng.uniform(0, grid, n)
    y = rng.uniform(0, grid, n)
    if shape == "corners":
        far = rng.integers(0, 2, n).astype(bool)
        x, y = np.where(far, grid - 2.0, 0.5) + 0.1 * rng.random(n), np.where(far, grid - 2.0, 0.5) + 0.1 * rng.random(n)
    elif shape == "one_cell":
        x, y = x * 0 + grid / 2 + 0.5, y * 0 + grid / 2 + 0.5
        D = 0.0
    elif shape == "end":
        y = grid - 1 + rng.random(n) * 0.9
    x, y = x.astype(np.float32), y.astype(np.float32)
    sp = rng.integers(0, 3, n).astype(np.uint8)
    p = ind.Particles(n, grid, D=D, vx=0.0, vy=0.0, dt=1.0, p_react=p_react, seed=seed)
    p.set(x, y, sp, step=0)
    p.step(1)
    gx, gy, gs = p.get()
    assert p.status() == 0
    start, count, keys, idx = p.bins()
    ox, oy, osp = x.copy(), y.copy(), sp.copy()
    m = oracle.orc().orc_particles_run(n, oracle.ptr(ox), oracle.ptr(oy), oracle.ptr(osp), grid, D, 0.0, 0.0, 1.0,
                                       p_react, seed, 0, 1)
    assert gx.size == m
    assert np.array_equal(gx, ox[:m]) and np.array_equal(gy, oy[:m]) and np.array_equal(gs, osp[:m])
    assert keys.size == n and np.all(np.diff(keys.astype(np.int64)) >= 0)
    want = np.bincount(keys, minlength=grid * grid)
    assert np.array_equal(count, want)
    assert np.array_equal(start, (np.cumsum(want) - want).astype(np.uint32))
    assert np.array_equal(np.sort(idx), np.arange(n, dtype=np.uint32))


@pytest.mark.parametrize("grid,n,p_react", [(1, 1000, 1.0), (3, 5001, 1.0), (64, 9000, 0.5), (2, 70_000, 1.0), (200, 90_000, 0.7)])
def test_many_steps_in_one_call(gpgmp, grid, n, p_react):
    """More steps than between two reads of the number of particles, down to none, one
    species or lists shorter than the launches made for them."""
    from inchman_b200 import individual as ind
    steps, seed = 37, 9
    rng = np.random.default_rng(4)
    x, y = (rng.uniform(0, grid, n).astype(np.float32) for _ in range(2))
    sp = (np.arange(n) % 2).astype(np.uint8)
    ox, oy, osp = x.copy(), y.copy(), sp.copy()
    p = ind.Particles(n, grid, D=0.5, vx=0.0, vy=0.1, dt=1.0, p_react=p_react, seed=seed)
    p.set(x, y, sp, step=0)
    p.step(steps)
    gx, gy, gs = p.get()
    assert p.status() == 0
    start, count, _, _ = p.bins()
    m = oracle.orc().orc_particles_run(n, oracle.ptr(ox), oracle.ptr(oy), oracle.ptr(osp), grid, 0.5, 0.0, 0.1, 1.0,
                                       p_react, seed, 0, steps)
    assert gx.size == m
    assert np.array_equal(gx, ox[:m]) and np.array_equal(gy, oy[:m]) and np.array_equal(gs, osp[:m])
    assert np.array_equal(start, (np.cumsum(count) - count).astype(np.uint32))
