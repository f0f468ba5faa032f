"""The f64 adjoint's two routes, steps recorded as they ran and steps re-run from a
checkpoint, give the same bits: over intervals, a tape with some of each, sweeps in a row
with steps between them, and after calls that send every step to the re-run."""
import numpy as np
import pytest

from helpers import assert_bits_equal
from physics_b200 import scenes

pytestmark = pytest.mark.gpu

DT = 0.0025


def _world(gpu, dims, seed=5):
    from physics_b200 import SphParams
    sc = scenes.dam_break(*dims, box=8.0, dt=DT, steps=0)
    p = SphParams.defaults()
    p.bounds_min, p.bounds_max = sc.bounds_min, sc.bounds_max
    rng = np.random.default_rng(seed)
    w = gpu.FluidWorld(p)
    w.add_particles(sc.pos, np.full(sc.n, sc.mass), vel=rng.normal(0.0, 0.2, sc.pos.shape))
    return w, rng.normal(size=sc.pos.shape), rng.normal(size=sc.pos.shape)


def _same(a, b, what):
    for k in ("pos", "vel"):
        assert_bits_equal(a[k], b[k], f"{what}: {k}")
    assert a["stiffness"] == b["stiffness"] and a["visc_k0"] == b["visc_k0"], what


def _rerun(w):
    w.vel = w.vel  # a field written while the tape is on: the sweep re-runs every step


@pytest.mark.parametrize("dims,steps,every", [((1, 1, 1), 3, 2), ((9, 7, 11), 1, 1), ((9, 7, 11), 7, 3),
                                              ((16, 16, 16), 6, 9), ((60, 60, 60), 6, 3)])
def test_recorded_steps_equal_rerun_steps(gpu, dims, steps, every):
    w, gx, gv = _world(gpu, dims)
    w.tape_begin(every)
    w.step(DT, steps)
    got = w.step_backward(gx, gv)
    end = w.pos
    _same(w.step_backward(gx, gv), got, "second sweep")
    assert_bits_equal(w.pos, end, "state after the sweeps")
    _rerun(w)
    _same(w.step_backward(gx, gv), got, "re-run")
    w.tape_clear()


def test_steps_between_sweeps_and_a_new_tape(gpu):
    a, gx, gv = _world(gpu, (10, 12, 9))
    b, _, _ = _world(gpu, (10, 12, 9))
    a.tape_begin(4)
    b.tape_begin(4)
    _rerun(b)
    for steps in (3, 2, 6):
        a.step(DT, steps)
        b.step(DT, steps)
        _same(a.step_backward(gx, gv), b.step_backward(gx, gv), f"{a.tape_steps} steps")
    a.tape_clear()
    a.tape_begin(2)
    b.tape_clear()
    b.tape_begin(5)
    a.step(DT, 5)
    b.step(DT, 5)
    _same(a.step_backward(gx, gv), b.step_backward(gx, gv), "a new tape")


def test_fields_and_parameters_set_while_recording(gpu):
    ref, gx, gv = _world(gpu, (10, 12, 9))
    ref.tape_begin(3)
    ref.step(DT, 8)
    want = ref.step_backward(gx, gv)
    # The sweep follows the checkpoints: a velocity set inside a segment is not seen by it.
    w, _, _ = _world(gpu, (10, 12, 9))
    w.tape_begin(8)
    w.step(DT, 5)
    w.vel = np.zeros_like(gx)
    w.step(DT, 3)
    _same(w.step_backward(gx, gv), want, "velocity set inside the segment")
    # Parameters changed after the steps: the sweep re-runs them with the new ones.
    w, _, _ = _world(gpu, (10, 12, 9))
    w.tape_begin(8)
    w.step(DT, 8)
    p = w.params
    p.stiffness = 300.0
    w.params = p
    fresh, _, _ = _world(gpu, (10, 12, 9))
    fresh.params = p
    fresh.tape_begin(8)
    fresh.step(DT, 8)
    _same(w.step_backward(gx, gv), fresh.step_backward(gx, gv), "parameters changed before the sweep")
