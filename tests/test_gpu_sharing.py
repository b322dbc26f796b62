"""Simulations that share the GPU: several threads that each run one, and runs
long enough to be launched in parts.  The results are the bits of a run alone
and of single substeps, and neither holds up the other."""

import threading
import time

import numpy as np
import pytest

from conftest import bump, kelvin_helmholtz

import finitevolumegpu_b200 as fv

pytestmark = pytest.mark.gpu

WALLS = {"reflective": 0x03030303, "periodic": 0x02020202, "mixed": 0x02020303}
CHAIN_CELLS = 1 << 26  # cell updates of one launch (kChainCells in fv_api.cu)


def make(ctx, scheme, nx, ny, bc=0x03030303):
    b = fv.BoundaryCondition(fv.BoundaryCondition.getTypes(bc))
    if scheme.startswith("EE2D"):
        return fv.SCHEMES[scheme](ctx, *kelvin_helmholtz(nx, ny), nx, ny, 1.0 / nx, 1.0 / ny, 0.0, 1.4,
                                  boundary_conditions=b)
    return fv.SCHEMES[scheme](ctx, *bump(nx, ny), nx, ny, 1.0, 0.9, 9.81, boundary_conditions=b)


def side_by_side(works):
    """Runs the callables on a thread each and returns the wall time of all."""
    start, errors = threading.Barrier(len(works) + 1), []

    def run(work):
        start.wait()
        try:
            work()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(w,)) for w in works]
    for t in threads:
        t.start()
    start.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
    return time.perf_counter() - t0


@pytest.mark.parametrize("walls", list(WALLS))
@pytest.mark.parametrize("scheme", list(fv.SCHEMES))
def test_simulations_on_threads_equal_simulations_alone(ctx, scheme, walls):
    """Last tiles one cell wide, a single tile, several waves; the CFL schedule
    (300 steps, three dt intervals) and a last step that is cut short."""
    sizes = [(61, 67), (125, 61), (241, 57), (2, 2), (300, 310), (97, 700)]
    alone = []
    for nx, ny in sizes:
        sim = make(ctx, scheme, nx, ny, WALLS[walls])
        t = 250.5 * float(sim.computeDt()) * 0.9
        sim.simulate(t)
        alone.append((t, sim.download(), sim.simSteps(), sim.simTime(), sim.computeDt()))
        del sim
    sims = [make(ctx, scheme, nx, ny, WALLS[walls]) for nx, ny in sizes]
    side_by_side([lambda s=s, t=a[0]: s.simulate(t) for s, a in zip(sims, alone)])
    for size, s, (t, q, nt, t1, dt) in zip(sizes, sims, alone):
        assert (s.simSteps(), s.simTime(), s.computeDt()) == (nt, t1, dt) or scheme == "WAF" and s.simSteps() == nt, size
        for v, (x, y) in enumerate(zip(s.download(), q)):
            assert np.array_equal(x, y, equal_nan=True), (scheme, walls, size, v)


@pytest.mark.parametrize("scheme", list(fv.SCHEMES))
def test_run_in_several_launches_equals_single_substeps(ctx, scheme):
    """A number of steps for which the last substep begins in one launch and
    ends in the next, and the dt and CFL minimum that it leaves."""
    nx, ny = 3001, 2503
    a, b = make(ctx, scheme, nx, ny, WALLS["mixed"]), make(ctx, scheme, nx, ny, WALLS["mixed"])
    info = a.tile_info()
    tiles = -(-nx // info["tile_w"]) * -(-ny // info["tile_h"])
    part = CHAIN_CELLS // (info["tile_w"] * info["tile_h"])
    steps = next(n for n in range(2, 100) if n * a.num_substeps * tiles > part
                 and 0 < (n * a.num_substeps * tiles) % part < tiles)
    dt = np.float32(a.computeDt() * np.float32(0.3))
    before = a.launches()
    a.simulate((steps - 0.5) * float(dt), dt)
    assert a.launches() - before >= 2 and a.simSteps() == steps
    t = 0.0
    for k in range(steps):
        d = np.float32(min(float(dt), (steps - 0.5) * float(dt) - t))
        t += float(d)
        for i in range(b.num_substeps):
            b.substep(d, i)
    for v, (x, y) in enumerate(zip(a.download(), b.download())):
        assert np.array_equal(x, y), (scheme, v)
    assert a.computeDt() == b.computeDt()


def test_one_substep_in_several_launches(ctx):
    """More cells than one launch takes."""
    nx = ny = 12001
    h = np.ones((ny, nx), np.float32)
    h[5000:5100, 11900:12000] = 1.5
    z = np.zeros((ny, nx), np.float32)
    a, b = (fv.LxF.LxF(ctx, h, z, z, nx, ny, 1.0, 1.0, 9.81) for _ in range(2))
    dt = np.float32(a.computeDt() * np.float32(0.4))
    a.simulate(3 * float(dt), dt)
    assert a.simSteps() == 3 and a.launches() >= 3
    for _ in range(3):
        b.substep(dt, 0)
    assert np.array_equal(a.u0[0].download(None), b.u0[0].download(None))
    assert a.computeDt() == b.computeDt()


def test_small_simulations_run_side_by_side(ctx):
    """Eight 256 x 256 simulations of 600 steps: a third of the time that they
    take one after the other, here less than two thirds."""
    sims = [make(ctx, "KP07_dimsplit", 256, 256) for _ in range(8)]
    dt = float(sims[0].computeDt()) * 0.3

    def run(s):
        for _ in range(6):
            s.simulate(99.5 * dt, dt)

    for s in sims:
        run(s)
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        for s in sims:
            run(s)
        serial = time.perf_counter() - t0
        times.append(side_by_side([lambda s=s: run(s) for s in sims]) / serial)
    assert min(times) < 2.0 / 3.0, times


def test_small_simulation_beside_a_large_one(ctx):
    """20 steps of 256 x 256, and one, wait for a part of the large grid's 100 steps only."""
    big, small = make(ctx, "KP07_dimsplit", 4096, 4096), make(ctx, "KP07_dimsplit", 256, 256)
    db, ds = float(big.computeDt()) * 0.3, float(small.computeDt()) * 0.3
    big.simulate(99.5 * db, db)
    t0 = time.perf_counter()
    big.simulate(99.5 * db, db)
    alone = time.perf_counter() - t0
    stop, waits, steps = threading.Event(), [], []

    def run_big():
        while not stop.is_set():
            big.simulate(99.5 * db, db)

    def run_small():
        time.sleep(0.05)
        for _ in range(10):
            t0 = time.perf_counter()
            small.simulate(19.5 * ds, ds)
            t1 = time.perf_counter()
            waits.append(t1 - t0)
            small.step(np.float32(ds))
            small.synchronize()
            steps.append(time.perf_counter() - t1)
        stop.set()

    side_by_side([run_big, run_small])
    assert sorted(waits)[5] < 0.3 * alone, (waits, alone)
    assert sorted(steps)[5] < 0.03 * alone, (steps, alone)


def test_steps_on_threads_equal_steps_alone(ctx):
    """step() with and without another simulation in the context."""
    nx, ny = 300, 310
    alone = make(ctx, "KP07_dimsplit", nx, ny)
    dt = np.float32(alone.computeDt() * np.float32(0.4))

    def run(s):
        for _ in range(40):
            s.step(dt)
        s.synchronize()

    run(alone)
    want = alone.download()
    sims = [make(ctx, "KP07_dimsplit", nx, ny) for _ in range(4)]
    side_by_side([lambda s=s: run(s) for s in sims])
    for s in sims:
        assert s.simSteps() == 40 and s.computeDt() == alone.computeDt()
        for x, y in zip(s.download(), want):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("dt", [None, np.inf, np.nan, 0.0, -1.0])
def test_advance_of_several_intervals_in_chains(ctx, dt):
    """advance() over three dt intervals on a grid whose runs are chains, against
    single steps of it; a dt that is not a positive number ends it after the
    step that it spoils, or before the first."""
    nx, ny = 1500, 1201
    a, b = make(ctx, "KP07_dimsplit", nx, ny), make(ctx, "KP07_dimsplit", nx, ny)
    if dt is None:
        a.advance(230)
        while b.simSteps() < 230:
            b.advance(1)
        assert a.simSteps() == b.simSteps() == 230 and a.simTime() == b.simTime()
        for x, y in zip(a.download(), b.download()):
            assert np.array_equal(x, y)
        return
    t, nt, _, cfl = a.get_control()
    a.set_control(t, 150, np.float32(dt), cfl)  # in the middle of an interval: this dt is used
    a.advance(200)
    assert a.simSteps() == (150 if dt <= 0.0 else 151)
    assert np.isfinite(a.simTime()) == (dt <= 0.0)
