"""A batch's steps give the same bits whether a run of them is one launch, over
all substeps, or each substep a launch of its own, with simulations that reach
their end or fail in the middle of a run."""

import numpy as np
import pytest

from conftest import bump, dam_break, kelvin_helmholtz

import finitevolumegpu_b200 as fv
from finitevolumegpu_b200.batch import Batch

pytestmark = pytest.mark.gpu

PERIODIC = fv.BoundaryCondition(fv.BoundaryCondition.getTypes(0x02020202))
STEPS = 400
SIZES = [(64, 64), (97, 150), (61, 130), (300, 70), (33, 200), (2, 2), (250, 250)]


def scenarios(scheme):
    """Uneven grids: ends after 1 to about 270 steps, one end time already reached."""
    for k, (nx, ny) in enumerate(SIZES):
        if scheme.startswith("EE2D"):
            q, dx, dy, unit = list(kelvin_helmholtz(nx, ny)), 1.0 / nx, 1.0 / ny, 1.0 / max(nx, ny)
        else:
            q, dx, dy, unit = list(bump(nx, ny) if k % 2 else dam_break(nx, ny)), 1.0, 0.9, 1.0
        yield q, nx, ny, dx, dy, (0.0 if k == 2 else 0.07 + 2.5 * k) * unit


def make(ctx, scheme, **kw):
    b = Batch(ctx, scheme, g=0.0 if scheme.startswith("EE2D") else 9.81, max_instances=16, cfl_scale=0.45, **kw)
    bc = PERIODIC if scheme.startswith("EE2D") else None
    slots = [b.add(q, nx, ny, dx, dy, t, bc) for q, nx, ny, dx, dy, t in scenarios(scheme)]
    return b, slots


@pytest.mark.parametrize("scheme", list(fv.SCHEMES))
def test_long_run_equals_single_steps_and_plain(ctx, scheme):
    a, slots = make(ctx, scheme)
    before = a.launches()
    a.run(STEPS)  # past every end
    assert a.launches() - before <= 4  # one run of 400 steps, in parts of 2^26 cell updates
    b, _ = make(ctx, scheme)
    for _ in range(STEPS):
        b.run(1)
    c, _ = make(ctx, scheme, shared=True)
    before = c.launches()
    c.run(STEPS)
    assert c.launches() - before == STEPS * (1 if scheme in ("LxF", "FORCE", "HLL") else 2)
    for batch in (a, b, c):
        batch.sync()
    for s, (q, nx, ny, dx, dy, t) in zip(slots, scenarios(scheme)):
        cls, kw = fv.SCHEMES[scheme], {"cfl_scale": 0.45}
        if scheme.startswith("EE2D"):
            sim = cls(ctx, *q, nx, ny, dx, dy, 0.0, 1.4, boundary_conditions=PERIODIC, **kw)
        else:
            sim = cls(ctx, *q, nx, ny, dx, dy, 9.81, **kw)
        sim.simulate(t)
        want = sim.download()
        for batch in (a, b, c):
            st = batch.status(s)
            assert st["done"] and not st["failed"] and (st["nt"], st["t"]) == (sim.simSteps(), sim.simTime()), (nx, ny)
            for x, y in zip(batch.download(s), want):
                assert np.array_equal(x, y, equal_nan=True), (scheme, nx, ny)


@pytest.mark.parametrize("scheme", ["HLL", "KP07", "KP07_dimsplit"])
def test_failures_in_the_middle_of_a_run(ctx, scheme):
    """A simulation whose state goes bad stops at that step, alone, in a run as in single steps."""
    def states(batch):
        out = []
        for k, (nx, ny) in enumerate([(90, 61), (130, 131), (64, 64), (61, 200)]):
            q = [a.copy() for a in bump(nx, ny)]
            if k in (1, 3):
                q[0][ny // 2, nx // 2] = np.nan if k == 1 else 1e-30
                q[1][ny // 2, nx // 2] = 50.0
            out.append(batch.add(q, nx, ny, 1.0, 1.0, 4.0))
        return out

    a, b = (Batch(ctx, scheme, max_instances=8) for _ in range(2))
    slots = states(a)
    states(b)
    a.run(60)
    for _ in range(60):
        b.run(1)
    a.sync()
    b.sync()
    assert {a.status(s)["failed"] for s in slots[1::2]} == {True} and not a.status(slots[0])["failed"]
    for s in slots:
        x, y = a.status(s), b.status(s)
        assert (x["nt"], x["failed"], x["done"]) == (y["nt"], y["failed"], y["done"])
        assert np.array_equal([x["t"], x["dt"]], [y["t"], y["dt"]], equal_nan=True)
        for u, v in zip(a.download(s), b.download(s)):
            assert np.array_equal(u, v, equal_nan=True)


def test_run_in_a_chain_of_launches(ctx):
    """More cell updates than one launch takes, and two batches at once, which take turns."""
    sizes = [(2048, 2048), (2000, 2050), (2048, 1990)]
    batches = [Batch(ctx, "KP07_dimsplit", max_instances=4) for _ in range(2)]
    sims = [fv.KP07_dimsplit.KP07_dimsplit(ctx, *bump(nx, ny), nx, ny, 1.0, 1.0, 9.81) for nx, ny in sizes]
    dts = [float(s.computeDt()) * 0.9 for s in sims]
    for b in batches:
        for (nx, ny), dt in zip(sizes, dts):
            b.add(list(bump(nx, ny)), nx, ny, 1.0, 1.0, 15.5 * dt)
    batches[0].run(20)
    assert 1 < batches[0].launches() < 40  # a run of 20 steps, 5e8 cell updates
    before = batches[1].launches()
    batches[1].run(20)
    assert batches[1].launches() - before == 40  # beside another one: a launch per substep
    for b in batches:
        b.sync()
    for k, (s, dt) in enumerate(zip(sims, dts)):
        s.simulate(15.5 * dt)
        for b in batches:
            assert b.status(k)["nt"] == s.simSteps()
            for x, y in zip(b.download(k), s.download()):
                assert np.array_equal(x, y)


def test_retired_tile_indices_are_accepted(ctx):
    """Indices 5 and 6 of KP07_dimsplit, which older timing caches may hold."""
    for old, now in ((5, 4), (6, 1)):
        a, b = (Batch(ctx, "KP07_dimsplit", tile=t, max_instances=2).info() for t in (old, now))
        assert [a[k] for k in ("tile_w", "tile_h", "threads")] == [b[k] for k in ("tile_w", "tile_h", "threads")]
