"""Rules by the number of cells or tiles that worlds of few particles meet: wide boxes take the
sort of several launches, few 2x2x2 tiles are split into x-slabs.  The same scene on both sides
of each rule gives the same bits."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho", "p", "acc", "xsph")


def _world(gpu, form, tile, top, pos, vel):
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (top,) * 3
    w = gpu.FluidWorld(p, form)
    if form == "comp":
        w.set_tuning(comp_tile=tile)
    w.add_particles(pos, scenes.lattice_mass(0.1), vel=vel)
    return w


@pytest.mark.parametrize("n", [1, 33, 3000])
@pytest.mark.parametrize("form,tile,wide", [("f64", 0, 40.0), ("comp", 0, 40.0), ("comp", 2, 66.0)])
def test_few_particles_in_a_wide_box(gpu, form, tile, wide, n):
    """8 million cells, or 4.5 million tiles, against a box of the particles' own size.  (No
    particle reaches a wall.)"""
    rng = np.random.default_rng(n)
    pos, vel = 1.0 + rng.uniform(0.0, 1.5, (n, 3)), rng.normal(0.0, 0.2, (n, 3))
    a, b = _world(gpu, form, tile, 4.0, pos, vel), _world(gpu, form, tile, wide, pos, vel)
    for w in (a, b):
        w.step(0.002, 4)
    for k in FIELDS:
        assert_bits_equal(getattr(a, k), getattr(b, k), k)


@pytest.mark.parametrize("n", [33, 5000, 70001])
@pytest.mark.parametrize("shuffled", [False, True])
def test_one_particle_per_cell(gpu, oracle_mod, n, shuffled):
    """The one-launch sort's scan sums where warps lie in one scan tile (4096 cells) and in several."""
    O = oracle_mod
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    i = rng.permutation(n) if shuffled else np.arange(n)
    pos = (np.stack([i // (m * m), (i // m) % m, i % m], axis=1) + 0.5) * 0.2 + rng.uniform(-0.09, 0.09, (n, 3))
    vel = rng.normal(0.0, 0.3, pos.shape)
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (0.2 * m,) * 3
    w, ow = gpu.FluidWorld(p), O.OracleWorld(p, threads=O.max_threads())
    for x in (w, ow):
        x.add_particles(pos, 1.0, vel=vel)
        x.step(0.002, 2)
    for name, f in (("pos", O.F_POS), ("vel", O.F_VEL), ("rho", O.F_RHO), ("acc", O.F_ACC)):
        assert_bits_equal(getattr(w, name), ow.get(f), name)
