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


@pytest.mark.parametrize("n,per_cell", [(33, 33), (700, 64), (6000, 160), (20000, 1100)])
@pytest.mark.parametrize("materials", [1, 3])
def test_dense_halves(gpu, oracle_mod, n, per_cell, materials):
    """Dense-cell tasks run in halves joined by the second to finish: sheets with one and many
    tasks per cell, kept masks and the filtering walk, against the oracle within the compensated
    form's bounds (density 1e-5; the sums of ~per_cell terms keep it far below) and twice for the
    same bits."""
    O = oracle_mod
    rng = np.random.default_rng(n)
    edge = 0.2 * max(1.0, n / per_cell) ** 0.5
    pos = rng.uniform(0.0, 1.0, (n, 3)) * [edge, 0.1, edge]
    vel = rng.normal(0.0, 0.1, (n, 3))
    mat = rng.integers(0, materials, n)
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (max(1.0, edge),) * 3
    if materials == 3:
        p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 0.7, 1.3]
    mass = scenes.lattice_mass(0.1)
    ow = O.OracleWorld(p, threads=O.max_threads())
    ow.add_particles(pos, mass, vel=vel, material=mat)
    ow.step(0.001)
    outs = []
    for masks in (1, 1, 0):
        w = gpu.FluidWorld(p, "comp")
        w.set_tuning(dense_masks=masks)
        w.add_particles(pos, mass, vel=vel, material=mat)
        w.step(0.001)
        w.synchronize()
        if masks:  # a second step from the same state finds the mask buffer grown
            w.set(gpu.FIELD_POS, pos)
            w.set(gpu.FIELD_VEL, vel)
            w.step(0.001)
        outs.append({k: getattr(w, k).copy() for k in FIELDS})
    for o in outs[1:]:
        for k in FIELDS:
            assert_bits_equal(o[k], outs[0][k], k)
    rho = ow.get(O.F_RHO)
    assert np.max(np.abs(outs[0]["rho"] - rho) / rho) <= 1e-5
    acc = ow.get(O.F_ACC)
    assert np.max(np.abs(outs[0]["acc"] - acc)) <= 1e-3 * np.max(np.abs(acc))
