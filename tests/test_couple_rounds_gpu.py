"""couple_heat's sort by source cell where the rounds per sort block change: one round
below and at 16,384 keys, two above it (the last block then holds one key), and the most
rounds. In-order sums, so the sources equal the oracle's bits."""
import numpy as np
import pytest

from helpers import assert_bits_equal, ref_test_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 257, 16383, 16384, 16385, 33000, 530001])
def test_heat_sources_at_the_edges_of_the_sort_blocks(gpu, oracle_mod, n):
    O = oracle_mod
    rng = np.random.default_rng(n)
    p = ref_test_params(gravity=(0.0, -9.81, 0.0))
    p.bounds_min, p.bounds_max = (-20.0,) * 3, (20.0,) * 3
    pos = rng.uniform(-9.0, 9.0, (n, 3))
    w = gpu.FluidWorld(p)
    w.add_particles(pos, 0.001)
    ow = O.OracleWorld(p, threads=O.max_threads())
    ow.add_particles(pos, np.full(n, 0.001))
    temp = rng.uniform(-1.0, 2.0, (21, 19, 23))
    src = rng.normal(0.0, 0.1, temp.shape)
    args = (0.01, 0.3, 0.2, 0.05)  # dt, t_ref, beta, heat_gain
    for origin in ((-10.0, -10.0, -10.0), (-3.0, -2.0, -4.0)):
        got = w.couple_heat(temp, src, origin, 1.0, *args)
        want = ow.couple_heat(temp, src, origin, 1.0, *args)
        assert_bits_equal(got, want, "sources")
        assert_bits_equal(w.body_acc, ow.get(O.F_BODY_ACC), "body accelerations")
        src = got


def test_one_point_in_memory_that_held_other_data(gpu, oracle_mod):
    """The words of couple_points' walk in a buffer that is not zero when it is allocated."""
    import torch
    O = oracle_mod
    for _ in range(4):
        dirty = [torch.full((1 << k,), -1, dtype=torch.int32, device="cuda") for k in range(7, 23)]
        torch.cuda.synchronize()
        del dirty
        torch.cuda.empty_cache()
        p = ref_test_params(gravity=(0.0, -9.81, 0.0))
        w, ow = gpu.FluidWorld(p), O.OracleWorld(p)
        for f in (w, ow):
            f.fill_box((-0.5,) * 3, (0.5,) * 3, 0.1, 0.05)
            f.step(0.0025, 2)
        args = (np.zeros((1, 3)), np.zeros((1, 3)), np.array([0.02]), 0.0025, 1.0, 1000.0)
        assert_bits_equal(w.couple_points(*args), ow.couple_points(*args), "forces")
        assert_bits_equal(w.vel, ow.get(O.F_VEL), "velocities")
