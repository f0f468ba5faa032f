"""Adjoint tapes that reuse a cleared tape's buffers against re-run ones and against worlds
without an earlier tape: the same bits."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

DT = 0.0025


def _world(gpu, dims, seed=5):
    sc = scenes.dam_break(*dims, box=8.0, dt=DT, steps=0)
    p = gpu.SphParams.defaults()
    p.bounds_min, p.bounds_max = sc.bounds_min, sc.bounds_max
    rng = np.random.default_rng(seed)
    w = gpu.FluidWorld(p)
    w.add_particles(sc.pos, np.full(sc.n, sc.mass), vel=rng.normal(0.0, 0.2, sc.pos.shape))
    return w, sc, rng


def _same(a, b, what):
    for k in ("pos", "vel"):
        assert_bits_equal(a[k], b[k], f"{what}: {k}")
    assert a["stiffness"] == b["stiffness"] and a["visc_k0"] == b["visc_k0"], what


def test_a_new_tape_recorded_and_rerun(gpu):
    """The second tape of one world records its steps as they run, the other's goes to the re-run."""
    a, sc, rng = _world(gpu, (10, 12, 9))
    b, _, _ = _world(gpu, (10, 12, 9))
    g = rng.normal(size=sc.pos.shape)
    for w in (a, b):
        w.tape_begin(4)
        w.step(DT, 3)
        w.step_backward(g, g)
        w.tape_clear()
        w.tape_begin(2)
        w.step(DT, 5)
    b.vel = b.vel  # a field written while the tape is on
    _same(a.step_backward(g, g), b.step_backward(g, g), "a new tape")


@pytest.mark.parametrize("more", [1, 40, 3000])
def test_a_tape_after_the_count_changed(gpu, more):
    """Particles added between two tapes (within and past the world's capacity): the second tape is
    that of a world without a first one."""
    a, sc, rng = _world(gpu, (10, 12, 9))
    b, _, _ = _world(gpu, (10, 12, 9))
    extra = rng.uniform(0.1, 1.0, (more, 3))
    g = rng.normal(size=(sc.n + more, 3))
    a.tape_begin(3)
    b_first = b.pos
    a.step(DT, 4)
    a.step_backward(g[:sc.n], None)
    a.tape_clear()
    a.set(gpu.FIELD_POS, b_first)
    a.set(gpu.FIELD_VEL, b.vel)
    for w in (a, b):
        w.add_particles(extra, sc.mass)
        w.tape_begin(3)
        w.step(DT, 7)
    _same(a.step_backward(g, g), b.step_backward(g, g), f"{more} more particles")
