"""The sort's tiles one per warp (many sparse tiles) against one per CTA: a scene alone in few
tiles and in a batch whose other scene brings thousands gives the same bits, on both sides of
the one-launch sort's limit."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho", "p", "acc", "xsph")


@pytest.mark.parametrize("tile", [4, 2])
@pytest.mark.parametrize("others", [20000, 90000])
@pytest.mark.parametrize("spread", [0.15, 0.5])
def test_warp_and_cta_tiles_give_the_same_bits(gpu, tile, others, spread):
    """The scene has tiles of one, of 31 to 33 and of hundreds of particles, and equal positions."""
    rng = np.random.default_rng(others + tile)
    n = 900
    edge = spread * n ** (1.0 / 3.0)
    pos = rng.uniform(0.0, edge, (n, 3))
    pos[:150] = 0.5 + rng.uniform(0.0, 0.15, (150, 3))  # a crowded cell
    for k, count in enumerate((31, 32, 33)):
        pos[150 + 40 * k:150 + 40 * k + count] = rng.uniform(0.02, 0.38, (count, 3)) + [0.8 * (k + 1), 0.0, 0.0]
    pos[400] = pos[401]
    vel = rng.normal(0.0, 0.3, pos.shape)
    top = max(4.0, edge + 0.5)
    wide = 0.9 * others ** (1.0 / 3.0)
    opos = rng.uniform(0.0, wide, (others, 3))
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (top,) * 3
    mass = scenes.lattice_mass(0.1)
    alone, both = gpu.FluidWorld(p, "comp"), gpu.FluidWorld(p, "comp")
    for w in (alone, both):
        w.set_tuning(comp_tile=tile)
    alone.add_particles(pos, mass, vel=vel)
    both.add_particles(np.concatenate([pos, opos]), mass, vel=np.concatenate([vel, np.zeros_like(opos)]))
    both.set_scenes([n, others], [(0.0,) * 3] * 2, [(top,) * 3, (wide,) * 3])
    for w in (alone, both):
        w.step(0.002, 3)
    for k in FIELDS:
        assert_bits_equal(getattr(alone, k), getattr(both, k)[:n], k)
