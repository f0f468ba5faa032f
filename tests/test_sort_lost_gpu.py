"""A step whose sort gives up at a grid barrier (sort_polls = 0: it never looks) does not
happen: the particles, their constants and the outputs stay as they were, the next wait reports
it once, and the world steps on as if it had not been asked."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import _lib as L
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

DT = 0.005
FIELDS = ("pos", "vel", "acc", "rho", "p", "xsph", "mass", "material", "body_acc")


def _world(gpu, form, tile, first_step=True, n=(11, 13, 9)):
    rng = np.random.default_rng(3)
    pos = scenes.dam_break_positions(*n)
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (3.0,) * 3
    p.visc_k, p.visc_n = [3.5, 2.0, 5.0], [1.0, 0.7, 1.3]
    w = gpu.FluidWorld(p, form)
    if form == "comp":
        w.set_tuning(comp_tile=tile)
    w.add_particles(pos, scenes.lattice_mass(0.1) * rng.uniform(0.9, 1.1, len(pos)),
                    vel=rng.normal(0.0, 0.3, pos.shape), material=rng.integers(0, 3, len(pos)))
    if first_step:
        w.step(DT, 2)
    return w, rng


def _state(w):
    return {k: getattr(w, k) for k in FIELDS}


@pytest.mark.parametrize("form,tile", [("f64", 0), ("comp", 4), ("comp", 2), ("comp", 0)])
@pytest.mark.parametrize("graph", [0, 3])
@pytest.mark.parametrize("first_step", [True, False])
def test_a_lost_step_does_not_happen(gpu, form, tile, graph, first_step):
    w, rng = _world(gpu, form, tile, first_step)
    ref, _ = _world(gpu, form, tile, first_step)
    push = rng.normal(0.0, 1.0, w.pos.shape)
    for v in (w, ref):
        v.set(gpu.FIELD_BODY_ACC, push)
    before = _state(w)
    w.set_tuning(sort_polls=0, graph_chunk=graph)
    w.step(DT, 4)
    with pytest.raises(L.PhyError, match="did not happen"):
        w.synchronize()
    for k, v in _state(w).items():
        assert_bits_equal(v, before[k], k)
    w.step(DT, 1)
    with pytest.raises(L.PhyError, match="did not happen"):
        w.get(gpu.FIELD_POS)
    w.set_tuning(sort_polls=1 << 22)
    w.step(DT, 5)
    ref.step(DT, 5)
    for k, v in _state(ref).items():
        assert_bits_equal(getattr(w, k), v, f"after {k}")


def test_a_lost_step_of_a_batch(gpu):
    batch = scenes.batch_scenes(4, 500, 3000, seed=2)
    pos = np.concatenate([b.pos for b in batch])
    p = gpu.SphParams.defaults()
    outs = []
    for polls in (0, 1 << 22):
        w = gpu.FluidWorld(p, "comp")
        w.add_particles(pos, scenes.lattice_mass(0.1))
        w.set_scenes([b.n for b in batch], [b.bounds_min for b in batch], [b.bounds_max for b in batch])
        w.set_tuning(sort_polls=polls)
        if polls == 0:
            w.step(DT, 3)
            with pytest.raises(L.PhyError, match="did not happen"):
                w.synchronize()
            w.set_tuning(sort_polls=1 << 22)
        w.step(DT, 3)
        outs.append(_state(w))
    for k in FIELDS:
        assert_bits_equal(outs[0][k], outs[1][k], k)


@pytest.mark.parametrize("form", ["f64", "comp"])
@pytest.mark.parametrize("when", ["recording", "sweeping"])
def test_a_tape_with_a_lost_step_is_not_swept(gpu, form, when):
    w, rng = _world(gpu, form, 4)
    g = rng.normal(size=w.pos.shape)
    w.tape_begin(2)
    w.step(DT, 2)
    w.set_tuning(sort_polls=0 if when == "recording" else 1 << 22)
    w.step(DT, 2)
    if when == "sweeping":
        w.vel = w.vel  # the sweep re-runs its steps
    w.set_tuning(sort_polls=0 if when == "sweeping" else 1 << 22)
    for _ in range(2):
        with pytest.raises(L.PhyError, match="did not happen"):
            w.step_backward(g, g)
    w.set_tuning(sort_polls=1 << 22)
    ref, _ = _world(gpu, form, 4)
    ref.set(gpu.FIELD_POS, w.pos)
    ref.set(gpu.FIELD_VEL, w.vel)
    out = []
    for v in (w, ref):
        v.tape_begin(2)
        v.step(DT, 3)
        out.append(v.step_backward(g, g))
    for k in ("pos", "vel"):
        assert_bits_equal(out[0][k], out[1][k], k)
