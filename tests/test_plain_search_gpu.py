"""The f64 step's neighbour search, packed pair operands and one-launch sort where they change
path: group edges, lanes per particle, the sort's size rule, crowded cells, spray, values outside
the reciprocals' safe range.  Bit for bit against the oracle."""
import numpy as np
import pytest

from helpers import assert_bits_equal

pytestmark = pytest.mark.gpu


def _random(rng, n, box, vel=0.3):
    return rng.uniform(0.0, 1.0, (n, 3)) * np.asarray(box), rng.normal(0.0, vel, (n, 3))


def _check(gpu, O, p, pos, vel, mass, material=None, steps=2, h=None, dt=0.0025):
    w, ow = gpu.FluidWorld(p), O.OracleWorld(p, threads=O.max_threads())
    w.add_particles(pos, mass, vel=vel, material=material)
    ow.add_particles(pos, mass, vel=vel, material=material)
    if h is not None:
        q = w.params
        q.h = h
        w.params = q
        ow.set_params(q)
    w.step(dt, steps)
    ow.step(dt, steps)
    for name, f in (("pos", O.F_POS), ("vel", O.F_VEL), ("rho", O.F_RHO), ("p", O.F_P), ("acc", O.F_ACC),
                    ("xsph", O.F_XSPH), ("mu_eff", O.F_MU_EFF)):
        assert_bits_equal(getattr(w, name), ow.get(f), name)


def _params(gpu, top, **over):
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0, 0.0, 0.0), (top, top, top)
    for k, v in over.items():
        setattr(p, k, v)
    return p


# One group short, full and over; a group of several columns; both lane counts of the force pass
# (below and above 16,384); both sides of the one-launch sort's 80,000.
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 16383, 16385, 79999, 80001])
def test_sizes(gpu, oracle_mod, n):
    rng = np.random.default_rng(n)
    edge = (n / 1000.0) ** (1.0 / 3.0) + 0.05
    pos, vel = _random(rng, n, (edge, edge, edge))
    _check(gpu, oracle_mod, _params(gpu, 2.0 * edge), pos, vel, np.full(n, 1.0))


# Cells of 20 (two batches of candidates), 70 (lists overflow, cells past the counting order) and 300
# (the search leaves the group to the walk; the bitonic order in the one-launch sort).
@pytest.mark.parametrize("per_cell,n", [(20, 3000), (70, 5000), (300, 6000)])
@pytest.mark.parametrize("materials", [1, 3])
def test_crowded(gpu, oracle_mod, per_cell, n, materials):
    rng = np.random.default_rng(per_cell)
    edge = 0.2 * (n / per_cell) ** (1.0 / 3.0)
    pos, vel = _random(rng, n, (edge, edge, edge))
    p = _params(gpu, 2.0)
    if materials == 3:
        p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 1.0, 1.0]
    _check(gpu, oracle_mod, p, pos, vel, np.full(n, 1.0), material=rng.integers(0, materials, n))


def test_spray_and_columns(gpu, oracle_mod):
    """Isolated particles, thin segments and a dense block in one world; particles out of the box."""
    rng = np.random.default_rng(5)
    a, _ = _random(rng, 1500, (6.0, 6.0, 6.0))
    b, _ = _random(rng, 4000, (0.8, 3.0, 1.1))
    pos = np.concatenate([a, b])[rng.permutation(5500)]
    _check(gpu, oracle_mod, _params(gpu, 6.0), pos, rng.normal(0.0, 4.0, pos.shape), np.full(5500, 1.0), dt=0.02)


@pytest.mark.parametrize("h", [0.13, 0.27])
def test_live_h(gpu, oracle_mod, h):
    """A cutoff above the cell size must not reach past the 27 cells; below, it cuts."""
    rng = np.random.default_rng(8)
    pos, vel = _random(rng, 4000, (1.6, 1.6, 1.6))
    _check(gpu, oracle_mod, _params(gpu, 3.0), pos, vel, np.full(4000, 1.0), h=h)


@pytest.mark.parametrize("case", ["tiny coordinate", "huge mass", "tiny mass", "zero mass", "nan", "coincident"])
def test_outside_the_safe_range(gpu, oracle_mod, case):
    """One particle outside the range where quotients come from reciprocals (every quotient of the
    step is then divided plainly), and distances of zero and NaN."""
    rng = np.random.default_rng(9)
    n = 2000
    pos, vel = _random(rng, n, (1.3, 1.3, 1.3))
    mass = np.full(n, 1.0)
    if case == "tiny coordinate":
        pos[:4] = [[1e-250, 0.5, 0.5], [3e-250, 0.5, 0.5], [0.5, 1e-300, 0.5], [0.5, 2e-300, 0.5]]
    elif case == "huge mass":
        mass[7] = 1e70
    elif case == "tiny mass":
        mass[7] = 1e-70
    elif case == "zero mass":
        mass[::3] = 0.0
    elif case == "nan":
        pos[11, 1] = np.nan
    else:
        pos[20:25] = pos[19]
    w, ow = gpu.FluidWorld(_params(gpu, 2.0)), oracle_mod.OracleWorld(_params(gpu, 2.0))
    for x in (w, ow):
        x.add_particles(pos, mass, vel=vel)
        x.step(0.0025, 2)
    for name, f in (("pos", oracle_mod.F_POS), ("vel", oracle_mod.F_VEL), ("rho", oracle_mod.F_RHO),
                    ("acc", oracle_mod.F_ACC)):
        a, b = getattr(w, name), ow.get(f)
        nan = np.isnan(a) & np.isnan(b)
        assert_bits_equal(np.where(nan, 0.0, a), np.where(nan, 0.0, b), f"{case} {name}")


def test_quotients_by_reciprocal(gpu, oracle_mod):
    """Pairs at every scale of separation and position: the quotients of the force sum (d / r and
    m m / rho) equal plain division, seen through the accelerations."""
    rng = np.random.default_rng(10)
    n = 6000
    centre = rng.uniform(0.3, 5.7, (n // 2, 3))
    d = rng.normal(0.0, 1.0, (n // 2, 3)) * (0.1 * 2.0 ** -rng.uniform(0.0, 40.0, (n // 2, 1)))
    pos = np.concatenate([centre, centre + d])
    mass = 2.0 ** rng.uniform(-20.0, 20.0, n)
    _check(gpu, oracle_mod, _params(gpu, 6.0), pos, rng.normal(0.0, 0.2, (n, 3)), mass, steps=1)


@pytest.mark.parametrize("n", [257, 20000, 90000])
def test_graph_chunks_change_no_bit(gpu, n):
    """Steps replayed as CUDA graphs: overlapped launches and the one-launch sort (and, past their
    sizes, the separate kernels) captured."""
    rng = np.random.default_rng(n)
    edge = (n / 1000.0) ** (1.0 / 3.0) + 0.05
    pos, vel = _random(rng, n, (edge, edge, edge))
    outs = []
    for chunk in (0, 3):
        w = gpu.FluidWorld(_params(gpu, 2.0 * edge))
        w.add_particles(pos, np.full(n, 1.0), vel=vel)
        w.set_tuning(graph_chunk=chunk)
        w.step(0.0025, 8)
        outs.append((w.pos, w.vel, w.acc))
    for a, b, name in zip(*outs, ("pos", "vel", "acc")):
        assert_bits_equal(b, a, name)
