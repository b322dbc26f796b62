"""Each bounded wait of the stage kernels ends by its own limit, says which it
was, and leaves the context usable: tile loads, neighbouring tiles in a run of
several substeps (a CTA per task and looping CTAs), and the earlier substeps of a
batch's simulation.  A limit of 0 polls gives up at once; nothing faults."""

import threading

import numpy as np
import pytest

from conftest import bump

import finitevolumegpu_b200 as fv
from finitevolumegpu_b200 import _lib
from finitevolumegpu_b200.batch import Batch

pytestmark = pytest.mark.gpu


def make(ctx, scheme="KP07_dimsplit", nx=300, ny=200):
    return fv.SCHEMES[scheme](ctx, *bump(nx, ny), nx, ny, 1.0, 1.0, 9.81)


def check_usable(ctx):
    a, b = make(ctx), make(ctx)
    dt = np.float32(a.computeDt() * np.float32(0.4))
    a.simulate(4 * float(dt), dt)
    for _ in range(a.simSteps()):
        for i in range(2):
            b.substep(dt, i)
    assert np.array_equal(a.download()[0], b.download()[0])


@pytest.mark.parametrize("scheme", ["LxF", "KP07_dimsplit"])
def test_neighbour_wait_has_its_own_limit(ctx, scheme):
    sim = make(ctx, scheme)
    _lib.check(_lib.lib().fv_sim_set_neighbour_wait_limit(sim._handle, 0))
    sim.substep(np.float32(0.01), 0)  # one substep waits for no neighbour
    sim.simSteps()
    with pytest.raises(_lib.FVError, match="gave up waiting for a neighbouring tile"):
        sim.simulate(2.0)
    del sim
    check_usable(ctx)


def test_tile_load_is_named(ctx):
    sim = make(ctx)
    _lib.check(_lib.lib().fv_sim_set_wait_limit(sim._handle, 0))
    sim.substep(np.float32(0.01), 0)
    with pytest.raises(_lib.FVError, match="gave up waiting for its tile load$"):
        sim.simSteps()
    del sim
    check_usable(ctx)


@pytest.mark.parametrize("neighbours", [True, False])
def test_looping_form_gives_up(ctx, neighbours):
    """Beside another simulation's run, CTAs loop over tasks: a wait that ran out
    does not stop them, and the other simulation is not affected."""
    bad, good, alone = make(ctx), make(ctx), make(ctx)
    dt = float(good.computeDt()) * 0.4
    f = _lib.lib().fv_sim_set_neighbour_wait_limit if neighbours else _lib.lib().fv_sim_set_wait_limit
    _lib.check(f(bad._handle, 0))
    started, errors = threading.Event(), []

    def run_good():
        for k in range(30):
            good.simulate(99.5 * dt, dt)
            started.set()

    t = threading.Thread(target=run_good)
    t.start()
    started.wait()
    try:
        bad.simulate(99.5 * dt, dt)
    except _lib.FVError as e:
        errors.append(str(e))
    t.join()
    assert errors and "gave up" in errors[0] and ("neighbouring" in errors[0] or not neighbours), errors
    for k in range(30):
        alone.simulate(99.5 * dt, dt)
    for x, y in zip(good.download(), alone.download()):
        assert np.array_equal(x, y)
    del bad
    check_usable(ctx)


def test_batch_wait_gives_up(ctx):
    def batch():
        b = Batch(ctx, "KP07_dimsplit", max_instances=8)
        for k in range(4):
            b.add(list(bump(100 + k, 90)), 100 + k, 90, 1.0, 1.0, 5.0)
        return b

    b = batch()
    _lib.check(_lib.lib().fv_batch_set_wait_limit(b._h, 0))
    b.run(1)  # a launch per substep waits for nothing
    b.sync()
    b.run(8)
    with pytest.raises(_lib.FVError, match="gave up waiting for an earlier substep"):
        b.sync()
    del b
    a, b = batch(), batch()
    _lib.check(_lib.lib().fv_batch_set_wait_limit(a._h, 0))
    _lib.check(_lib.lib().fv_batch_set_wait_limit(a._h, -1))
    a.run_to_completion()
    b.run_to_completion()
    for s in range(4):
        assert np.array_equal(a.download(s)[0], b.download(s)[0])
