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
