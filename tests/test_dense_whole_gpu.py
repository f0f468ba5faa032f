"""Dense-cell tasks by halves (worlds below 200,000 particles) and whole (from there on) give the
same bits, and the sums are the oracle's within what f32 terms allow."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "rho", "p", "acc", "xsph", "mu_eff")


def _sheet(rng, n, per_cell):
    edge = 0.2 * max(1.0, n / per_cell) ** 0.5
    return rng.uniform(0.0, 1.0, (n, 3)) * [edge, 0.1, edge], max(1.0, edge)


def _params(gpu, top, materials):
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (top,) * 3
    if materials == 3:
        p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 0.7, 1.3]
    return p


@pytest.mark.parametrize("n,per_cell", [(33, 33), (40, 40), (700, 64), (6000, 160), (20000, 1100)])
@pytest.mark.parametrize("materials", [1, 3])
@pytest.mark.parametrize("masks", [0, 1])
@pytest.mark.parametrize("tile", [4, 2])
def test_halves_and_whole_tasks_give_the_same_bits(gpu, n, per_cell, materials, masks, tile):
    """Alone by halves, and in a batch of 200,000 and more whole: with the kept masks (the second
    round of steps, when their buffer has grown) and filtering again."""
    rng = np.random.default_rng(n)
    pos, top = _sheet(rng, n, per_cell)
    others = 201000
    opos = scenes.dam_break_positions(60, 60, 56)[:others]
    vel, mat = rng.normal(0.0, 0.1, pos.shape), rng.integers(0, materials, n)
    p = _params(gpu, top, materials)
    mass = scenes.lattice_mass(0.1)
    alone, both = gpu.FluidWorld(p, "comp"), gpu.FluidWorld(p, "comp")
    allpos, allvel = np.concatenate([pos, opos]), np.concatenate([vel, np.zeros_like(opos)])
    for w in (alone, both):
        w.set_tuning(comp_tile=tile, dense_masks=masks)
    alone.add_particles(pos, mass, vel=vel, material=mat)
    both.add_particles(allpos, mass, vel=allvel, material=np.concatenate([mat, np.zeros(len(opos), np.int64)]))
    both.set_scenes([n, len(opos)], [(0.0,) * 3] * 2, [(top,) * 3, (12.0,) * 3])
    for start in (0, 1):
        for w, x, v in ((alone, pos, vel), (both, allpos, allvel)):
            if start:
                w.set(gpu.FIELD_POS, x)
                w.set(gpu.FIELD_VEL, v)
            w.step(0.001, 2)
            w.synchronize()
        for k in FIELDS:
            assert_bits_equal(getattr(alone, k), getattr(both, k)[:n], k)


@pytest.mark.parametrize("n,per_cell", [(33, 33), (700, 64), (5000, 160), (6000, 1100)])
@pytest.mark.parametrize("whole", [False, True])
def test_dense_sums_against_the_terms(gpu, n, per_cell, whole):
    """Density, acceleration and XSPH of a sheet of one material against 64-bit sums over all pairs.
    A pair term takes some 20 roundings of 2^-24 (1.2e-6 of it), and the cell-local coordinates'
    2^-25 of a cell change a term at the typical distance by less: 1e-5 of the summed absolute
    terms bounds the error, and a lost or doubled half exceeds it many times."""
    import torch
    rng = np.random.default_rng(n)
    pos, top = _sheet(rng, n, per_cell)
    vel = rng.normal(0.0, 0.1, pos.shape)
    p = _params(gpu, top, 1)
    mass = scenes.lattice_mass(0.1)
    w = gpu.FluidWorld(p, "comp")
    if whole:
        opos = scenes.dam_break_positions(60, 60, 56)
        w.add_particles(np.concatenate([pos, opos]), mass, vel=np.concatenate([vel, np.zeros_like(opos)]))
        w.set_scenes([n, len(opos)], [(0.0,) * 3] * 2, [(top,) * 3, (12.0,) * 3])
    else:
        w.add_particles(pos, mass, vel=vel)
    w.step(0.001)
    got = {k: torch.from_numpy(getattr(w, k)[:n]) for k in ("rho", "acc", "xsph")}

    h, m = 0.2, mass
    c6, cs, cl = 315.0 / (64.0 * np.pi * h ** 9), -45.0 / (np.pi * h ** 6), 45.0 / (np.pi * h ** 6)
    x, v = torch.from_numpy(pos), torch.from_numpy(vel)
    d = x[None] - x[:, None]
    r = d.norm(dim=2)
    near = r < h
    w6 = torch.where(near, c6 * (h * h - r * r) ** 3, 0.0)
    rho = m * w6.sum(1)
    assert ((got["rho"] - rho).abs() <= 1e-5 * rho).all()
    pr = p.stiffness * torch.clamp(rho - p.rest_density, min=0.0)
    pr2, mr = pr / rho ** 2, m / rho
    pair = near & (r > 0)
    dv = v[None] - v[:, None]
    xw = torch.where(pair, w6 * mr[None], 0.0)
    xs, xs_abs = (dv * xw[..., None]).sum(1), (dv.abs() * xw[..., None]).sum(1)
    assert ((got["xsph"] - xs).abs() <= 1e-5 * xs_abs + 1e-12).all()
    fp = torch.where(pair, m * m * (pr2[:, None] + pr2[None]) * cs * (h - r) ** 2 / torch.where(pair, r, 1.0), 0.0)
    fv = torch.where(pair, m * mr[None] * cl * (h - r), 0.0)
    mu = p.visc_k[0]
    acc = ((d * fp[..., None]).sum(1) + (dv * fv[..., None]).sum(1) * mu) / rho[:, None]
    size = ((d.abs() * fp.abs()[..., None]).sum(1) + (dv.abs() * fv[..., None]).sum(1) * mu) / rho[:, None]
    assert ((got["acc"] - acc).abs() <= 1e-5 * size + 1e-9).all()


def test_long_tasks_of_a_large_world(gpu):
    """300 particles per cell: whole tasks until the reservations are known, halves from then on."""
    n = 200003
    rng = np.random.default_rng(n)
    pos, top = _sheet(rng, n, 300)
    vel = rng.normal(0.0, 0.1, pos.shape)
    w = gpu.FluidWorld(_params(gpu, top, 1), "comp")
    w.add_particles(pos, scenes.lattice_mass(0.1), vel=vel)
    outs = []
    for start in range(3):
        if start:
            w.set(gpu.FIELD_POS, pos)
            w.set(gpu.FIELD_VEL, vel)
        w.step(0.001)
        outs.append({k: getattr(w, k).copy() for k in FIELDS})
        assert w.dense_mask_info()["demand"] > 1.5 * n
    for o in outs[1:]:
        for k in FIELDS:
            assert_bits_equal(o[k], outs[0][k], k)
