"""The library's host side on a CUDA runtime without a GPU (fake_cudart.cpp): what it
allocates, copies, refuses and reports.  Kernels do nothing there, so no values are compared."""
import ctypes as C
import gc
import importlib.util
import subprocess
from pathlib import Path

import numpy as np
import pytest

import physics_b200 as pb
from physics_b200 import _lib as L

ROOT = Path(__file__).resolve().parent.parent
DT = 0.0025


@pytest.fixture(scope="session")
def fake_library(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("phy_build", ROOT / "physics_b200" / "csrc" / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    try:
        cuda = Path(build._nvcc()).parents[1] / "include"
    except RuntimeError as e:
        pytest.skip(str(e))
    build.build_product()
    out = tmp_path_factory.mktemp("fake") / "libphysph_fake.so"
    objs = [build.OBJDIR / (s + ".o") for s in build.SOURCES]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", cuda, "-Wl,-Bsymbolic",
                    ROOT / "tests" / "fake_cudart.cpp", *objs, "-o", out, "-lpthread", "-ldl"], check=True)
    lib = C.CDLL(str(out))
    for name, (res, args) in L.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_live.restype = C.c_ulonglong
    lib.fake_set_budget.argtypes = [C.c_ulonglong]
    lib.fake_poke_pinned.argtypes = [C.c_ulonglong, C.c_ulonglong, C.c_uint32]
    lib.fake_launches.argtypes = [C.c_char_p]
    return lib


@pytest.fixture
def fake(fake_library, monkeypatch):
    monkeypatch.setattr(L, "_lib", fake_library)
    fake_library.fake_reset()
    yield fake_library
    for o in gc.get_objects():  # worlds go before the library is switched back
        if isinstance(o, pb.World):
            o.close()


def _world(form="f64", n=64, **kw):
    p = pb.SphParams.defaults()
    p.bounds_min, p.bounds_max = (0.0,) * 3, (2.0,) * 3
    w = pb.FluidWorld(p, form)
    w.add_particles(np.random.default_rng(n).uniform(0.1, 1.9, (n, 3)), 0.02, **kw)
    return w


@pytest.mark.parametrize("form", ["f64", "comp"])
@pytest.mark.parametrize("swept", [False, True])
def test_particles_added_while_a_tape_records(fake, form, swept):
    """The world takes them and steps on; the tape, whose checkpoints hold the old ones, is not
    swept any more, and no buffer sized for them is written past its end."""
    w = _world(form)
    w.tape_begin(2)
    w.step(DT, 3)
    g = np.ones((64, 3))
    if swept:
        w.step_backward(g, g)
    w.add_particles(np.full((200, 3), 0.5), 0.02)
    w.step(DT, 6)
    assert len(w) == 264 and w.tape_steps == 9
    g = np.ones((264, 3))
    with pytest.raises(L.PhyError, match="particles were added"):
        w.step_backward(g, g)
    assert fake.fake_violations() == 0
    w.tape_clear()
    w.tape_begin(2)
    w.step(DT, 3)
    w.step_backward(g, g)
    assert fake.fake_violations() == 0


def test_particles_added_to_a_tape_without_steps(fake):
    """Nothing to sweep: the seeds are the gradients, as for any such tape."""
    w = _world()
    w.tape_begin(2)
    w.step(DT, 2)
    w.step_backward(np.ones((64, 3)), None)
    w.tape_begin(2)
    w.add_particles(np.full((200, 3), 0.5), 0.02)
    w.step_backward(np.ones((264, 3)), None)
    assert fake.fake_violations() == 0


def test_failed_allocations_leave_no_stale_capacity(fake):
    """A scene table, a grid or a particle array that could not be had: the call fails, and the
    next one that fits an earlier capacity allocates instead of using what is gone."""
    w = _world("comp")
    w.set_scenes([32, 32], [(0.0,) * 3] * 2, [(2.0,) * 3] * 2)
    w.step(DT)
    w.clear_scenes()
    fake.fake_set_budget(fake.fake_live())
    counts = [64] + [0] * 3999
    with pytest.raises(L.PhyError, match="out of memory"):
        w.set_scenes(counts, [(0.0,) * 3] * 4000, [(0.1,) * 3] * 4000)
    fake.fake_set_budget(1 << 40)
    w.set_scenes([32, 32], [(0.0,) * 3] * 2, [(2.0,) * 3] * 2)
    w.step(DT)
    fake.fake_set_budget(fake.fake_live() + (1 << 19))  # room for the table of scenes, not for their boxes
    with pytest.raises(L.PhyError, match="out of memory"):
        w.set_scenes(counts, [(0.0,) * 3] * 4000, [(0.1,) * 3] * 4000)
        w.step(DT)
    fake.fake_set_budget(1 << 40)
    w.set(pb.FIELD_POS, np.full((64, 3), 0.5))
    w.clear_scenes()
    w.set_scenes([32, 32], [(0.0,) * 3] * 2, [(2.0,) * 3] * 2)
    w.step(DT)
    assert fake.fake_violations() == 0


@pytest.mark.parametrize("form", ["f64", "comp"])
@pytest.mark.parametrize("room", [0.2, 0.5, 0.8, 0.95])
def test_a_growth_that_fails_is_made_up_for(fake, form, room):
    """add_particles fails part way through the growth: the world steps on with what it had,
    allocating the arrays that the attempt gave up."""
    sizes = []
    for n in (64, 64 + 20000):
        w = _world(form, n=n)
        w.step(DT)
        sizes.append(fake.fake_live())
        w._world.close()
    w = _world(form)
    w.step(DT)
    fake.fake_set_budget(int(fake.fake_live() + room * (sizes[1] - sizes[0])))
    with pytest.raises(L.PhyError, match="out of memory"):
        w.add_particles(np.full((20000, 3), 0.5), 0.02)
    fake.fake_set_budget(1 << 40)
    calls = fake.fake_device_calls()
    w.step(DT)
    # (The first fifth of the memory goes to arrays that keep their old ones until then.)
    assert len(w) == 64 and (fake.fake_device_calls() > calls) == (room > 0.2)
    w.add_particles(np.full((20000, 3), 0.5), 0.02)
    w.step(DT)
    assert fake.fake_violations() == 0


def test_worlds_on_a_second_device(fake):
    """An f64 world on another device of the process after one on the first: the one-launch
    sort's shared-memory limit is set on each."""
    for device in (0, 1):
        fake.fake_set_device(device)
        w = _world()
        w.step(DT, 2)
        w.synchronize()
    assert fake.fake_launches(b"k_sort_fused") == 4


@pytest.mark.parametrize("form,most", [("f64", 42), ("comp", 59)])
def test_a_new_world_maps_few_blocks_of_memory(fake, form, most):
    """Creating a world, adding its particles and the first step: device allocations (each a
    block to map) no more than before the forms got further buffers, one page-locked one."""
    w = _world(form, n=64000)
    w.step(DT)
    assert fake.fake_device_calls() <= most and fake.fake_pinned_calls() <= 1


def test_a_lost_sort_is_reported_once_at_the_next_wait(fake):
    """The word a kernel sets in mapped memory (after the box and the mask demand)."""
    w = _world()
    for wait in (w.synchronize, lambda: w.get(pb.FIELD_RHO), lambda: w.pos, lambda: w.total_momentum()):
        w.step(DT)
        fake.fake_poke_pinned(64, 128, 1)
        with pytest.raises(L.PhyError, match="did not happen"):
            wait()
        wait()
    fake.fake_poke_pinned(64, 128, 1)
    with pytest.raises(L.PhyError, match="did not happen"):
        w._world.step_checked(DT)
    assert w._world.step_checked(DT) == 0
    w.tape_begin(2)
    w.step(DT, 3)
    fake.fake_poke_pinned(64, 128, 1)
    for _ in range(2):
        with pytest.raises(L.PhyError, match="did not happen"):
            w.step_backward(np.ones((64, 3)), None)
    w.tape_begin(2)
    w.step(DT, 3)
    w.step_backward(np.ones((64, 3)), None)


def _tape_world(n=4000):
    return _world(n=n), (22 * 8 + 99 * 4) * n, 48 * n  # one recorded step, one checkpoint


def test_recorded_steps_make_room_for_checkpoints(fake):
    """Steps recorded as they run fill the device; the checkpoints that the sweep cannot do
    without still find room, as they did while nothing was recorded."""
    w, slot, ckpt = _tape_world()
    w.step(DT)
    fake.fake_set_budget(int(fake.fake_live() + 4 * slot + 8 * ckpt))
    w.tape_begin(1)
    w.step(DT, 30)
    assert fake.fake_refused() > 0
    fake.fake_set_budget(1 << 40)
    w.step_backward(np.ones((4000, 3)), None)


def test_recorded_steps_make_room_for_the_sweep(fake):
    w, slot, ckpt = _tape_world()
    w.step(DT)
    fake.fake_set_budget(int(fake.fake_live() + 6.5 * slot))
    w.tape_begin(4)
    w.step(DT, 16)
    recorded = fake.fake_launches(b"k_tape_copy")
    w.step_backward(np.ones((4000, 3)), None)
    assert 0 < recorded < 16 and fake.fake_launches(b"k_tape_copy") >= recorded + 16


def test_a_cleared_tape_makes_room_for_the_world(fake):
    w, slot, ckpt = _tape_world()
    w.step(DT)
    before = fake.fake_live()
    w.tape_begin(5)
    w.step(DT, 10)
    w.step_backward(np.ones((4000, 3)), None)
    w.tape_clear()
    kept = fake.fake_live() - before
    assert kept > 8 * slot
    fake.fake_set_budget(fake.fake_live())
    w.set(pb.FIELD_BODY_ACC, np.ones((4000, 3)))
    assert fake.fake_live() < before + kept // 2
    fake.fake_set_budget(1 << 40)


def test_worlds_share_page_locked_memory(fake):
    """64 worlds a page; worlds made and dropped one after another lock no page each."""
    worlds = [_world() for _ in range(130)]
    assert fake.fake_pinned_calls() <= 3
    for w in worlds:
        w._world.close()
    for _ in range(5):
        _world()._world.close()
    assert fake.fake_pinned_calls() <= 3


@pytest.mark.parametrize("n,blocks", [(2000, {256}), (90000, {128, 256})])
@pytest.mark.parametrize("form", ["f64", "comp"])
def test_autotune_tries_the_sort_block_where_it_matters(fake, form, n, blocks):
    """Below 80,000 particles the sort is one launch without the knob: its values would time the
    same step twice."""
    trials = _world(form, n=n).autotune(DT, 1)
    assert {t["sort_block"] for t in trials} == blocks
    keys = [(t["comp_tile"], t["queue"], t["ctas_per_sm"], t["sort_block"]) for t in trials]
    assert len(set(keys)) == len(keys) >= len(blocks)


@pytest.mark.parametrize("form", ["f64", "comp"])
@pytest.mark.parametrize("n", [1, 300, 2000, 10000, 70000])
def test_the_one_launch_sort_leaves_room_for_other_worlds(fake, form, n):
    """A cooperative launch starts when all its blocks fit: one per 256 particles, or per SM where
    sparse tiles need them, not every one that the GPU (296 here) holds."""
    w = _world(form, n=n)
    w.step(DT)
    assert 1 <= fake.fake_cooperative_blocks() <= max(148, (n + 255) // 256)


@pytest.mark.parametrize("form", ["f64", "comp"])
def test_the_first_step_of_a_loaded_world_allocates_nothing(fake, form):
    w = _world(form, n=64000)
    calls = fake.fake_device_calls()
    w.step(DT)
    assert fake.fake_device_calls() == calls
