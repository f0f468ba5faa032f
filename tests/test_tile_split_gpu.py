"""The tiled passes' split of a tile into x-slabs (worlds of few tiles): the same scene stepped
with 4, 2 and 1 work items per tile gives the same bits."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho", "p", "acc", "xsph")


@pytest.mark.parametrize("dims", [(9, 11, 13), (30, 30, 30), (44, 60, 44)])
@pytest.mark.parametrize("materials", [1, 3])
def test_split_changes_no_bit(gpu, dims, materials):
    """Alone (under 150 tiles: 4 items each; under 600: 2) and in a batch whose other scene brings
    the tiles above both limits (1 item)."""
    rng = np.random.default_rng(sum(dims))
    pos = scenes.dam_break_positions(*dims)
    other = scenes.dam_break_positions(56, 100, 56)
    vel, ovel = rng.normal(0.0, 0.3, pos.shape), np.zeros_like(other)
    mat, omat = rng.integers(0, materials, len(pos)), np.zeros(len(other), np.int64)
    p = gpu.SphParams.defaults()
    top = 2.0 * max(dims) * 0.1
    p.bounds_min, p.bounds_max = (0.0,) * 3, (top,) * 3
    if materials == 3:
        p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 0.7, 1.3]
    mass = scenes.lattice_mass(0.1)
    alone = gpu.FluidWorld(p, "comp")
    alone.add_particles(pos, mass, vel=vel, material=mat)
    both = gpu.FluidWorld(p, "comp")
    both.add_particles(np.concatenate([pos, other]), mass, vel=np.concatenate([vel, ovel]),
                       material=np.concatenate([mat, omat]))
    both.set_scenes([len(pos), len(other)], [(0.0,) * 3] * 2, [(top,) * 3, (20.0,) * 3])
    for w in (alone, both):
        w.step(0.005, 3)
    for k in FIELDS:
        assert_bits_equal(getattr(alone, k), getattr(both, k)[:len(pos)], k)
