"""couple_points' walk against the oracle where its waits matter: a chain of points that
overlap only their neighbours, with more points than the GPU holds warps of the walk."""
import numpy as np
import pytest

from helpers import assert_bits_equal, ref_test_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,per_cell", [(6001, 2), (300, 40)])
def test_chain_of_overlapping_neighbours(gpu, oracle_mod, points, per_cell):
    """Points two cells (0.4) apart on a line: each reads the velocities that the one before it
    left in the cell they share, so a wait that orders too little shows in the bits."""
    O = oracle_mod
    rng = np.random.default_rng(points)
    length = 0.4 * (points + 2)
    n = int(length / 0.2) * per_cell
    pos = rng.uniform(0.0, 1.0, (n, 3)) * [length, 0.2, 0.2]
    vel = rng.normal(0.0, 0.5, (n, 3))
    p = ref_test_params(gravity=(0.0, -9.81, 0.0))
    p.bounds_min, p.bounds_max = (0.0,) * 3, (length, 0.2, 0.2)
    ppos = np.stack([0.4 * np.arange(1, points + 1) + 0.1, np.full(points, 0.1), np.full(points, 0.1)], axis=1)
    pvel = rng.normal(0.0, 0.5, (points, 3))
    mass = rng.uniform(0.01, 0.05, points)
    w, ow = gpu.FluidWorld(p), O.OracleWorld(p)
    for f in (w, ow):
        f.add_particles(pos, np.full(n, 0.02), vel=vel)
    args = (ppos, pvel, mass, 0.0025, 1.0, 1000.0)
    for _ in range(3):
        assert_bits_equal(w.couple_points(*args), ow.couple_points(*args), "forces")
        assert_bits_equal(w.vel, ow.get(O.F_VEL), "velocities")


def test_chain_of_heavy_points(gpu, oracle_mod):
    """40 points over the same 540,000 particles: each takes ~25 ms, so the last waits for a
    second; a wait's limit counts from the last point that was finished."""
    O = oracle_mod
    rng = np.random.default_rng(1)
    n, points = 27 * 20000, 40
    cell = np.arange(n) % 27
    pos = (np.stack([cell // 9, (cell // 3) % 3, cell % 3], axis=1) + rng.uniform(0.01, 0.99, (n, 3))) * 0.2
    vel = rng.normal(size=(n, 3))
    p = ref_test_params(gravity=(0.0, -9.81, 0.0))
    p.bounds_min, p.bounds_max = (0.0,) * 3, (0.6,) * 3
    args = (np.full((points, 3), 0.3), np.zeros((points, 3)), np.full(points, 0.02), 0.001, 1.0, 1000.0)
    w, ow = gpu.FluidWorld(p), O.OracleWorld(p)
    for f in (w, ow):
        f.add_particles(pos, np.full(n, 1e-4), vel=vel)
    assert_bits_equal(w.couple_points(*args), ow.couple_points(*args), "forces")
    assert_bits_equal(w.vel, ow.get(O.F_VEL), "velocities")
