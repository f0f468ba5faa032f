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


@pytest.mark.parametrize("dims", [(7, 8, 9), (16, 16, 16), (24, 30, 24)])
def test_split_of_small_tiles(gpu, dims):
    """2x2x2 tiles: alone (under 150 and under 600 of them) and beside a scene of thousands."""
    rng = np.random.default_rng(sum(dims))
    pos, other = scenes.dam_break_positions(*dims), scenes.dam_break_positions(40, 60, 40)
    vel = rng.normal(0.0, 0.3, pos.shape)
    top = 0.2 * max(dims)
    a = _world(gpu, "comp", 2, top, pos, vel)
    b = _world(gpu, "comp", 2, top, np.concatenate([pos, other]), np.concatenate([vel, np.zeros_like(other)]))
    b.set_scenes([len(pos), len(other)], [(0.0,) * 3] * 2, [(top,) * 3, (20.0,) * 3])
    for w in (a, b):
        w.step(0.005, 3)
    for k in FIELDS:
        assert_bits_equal(getattr(a, k), getattr(b, k)[:len(pos)], k)


@pytest.mark.parametrize("ns,per,flat", [(20, 3000, 0.1), (290, 200, 0.05), (290, 500, 1.0)])
def test_split_of_scenes_that_end_inside_a_tile(gpu, ns, per, flat):
    """Batches on both sides of the split's rules, the first and the last scene against a world of
    their own."""
    rng = np.random.default_rng(ns + per)
    m = int(np.ceil(per ** (1.0 / 3.0)))
    i = np.arange(per)
    one = (np.stack([i // (m * m), (i // m) % m, i % m], axis=1) + 0.5) * [0.1, 0.1 * flat, 0.1]
    pos = np.concatenate([one + rng.uniform(-0.002, 0.002, one.shape) for _ in range(ns)])
    vel = rng.normal(0.0, 0.1, pos.shape)
    both = _world(gpu, "comp", 4, 4.0, pos, vel)
    both.set_scenes([per] * ns, [(0.0,) * 3] * ns, [(4.0,) * 3] * ns)
    both.step(0.001, 2)
    for k in (0, ns - 1):
        part = slice(k * per, (k + 1) * per)
        alone = _world(gpu, "comp", 4, 4.0, pos[part], vel[part])
        alone.step(0.001, 2)
        for f in FIELDS:
            assert_bits_equal(getattr(alone, f), getattr(both, f)[part], f)


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
