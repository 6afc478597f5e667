"""Near lists (csrc/af3d_near.cu): a run that keeps them for up to 16 steps equals, bit for bit, one
whose every step starts from an import (which drops the lists, so that step's are new), whatever
the clumps' speed: within their allowances, past them (the clumps around search their cells)
and more than a cell per period (they search their flume).  For one flume and an ensemble, both
FP64 modes and phases, odd counts, and with a clump of more near pairs than a list holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 24


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


def wide_grid(af3d, g, margin):
    """The grid g widened by whole cells on every side."""
    g = g.copy()
    side = g["cell_side"]
    k = np.ceil(margin / side).astype(np.int64)
    g["rr_min"] -= k * side
    g["rr_max"] += k * side
    g["ncell"] += 2 * k
    g["length"] = g["rr_max"] - g["rr_min"]
    g["ncell3"] = int(np.prod(g["ncell"]))
    g["ntot"] = g["ncell3"] * g["ntags"]
    return g


def start(af3d, sys, fun, pp, mode, phase, speed, nflumes):
    """A context past its first re-grid, on a grid wide enough for the run."""
    e = af3d.Engine(sys, fun, ntags=0, fp_mode=mode, phase=phase)
    still = pp.copy()
    still["vv"] = 0.0
    still["ww"] = 0.0
    e.import_particles(still)
    e.step(1)
    for f in range(nflumes):
        e.set_flume_grid(f, wide_grid(af3d, e.get_flume_grid(f), 1.0 + 2.0 * speed * 2e-6 * STEPS))
    e.import_particles(pp)
    e.forces()
    e.swap_accel()
    return e


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("speed,n,nflumes,phase", [(20.0, 601, 1, 1), (3000.0, 601, 1, 1), (60000.0, 601, 1, 1),
                                                   (3000.0, 257, 2, 1), (60000.0, 129, 2, 1), (2000.0, 300, 1, 0)])
def test_kept_lists_equal_new_ones(af3d, mode, speed, n, nflumes, phase):
    from tests.states import flume_system, wall_state
    sys, fun = flume_system(n, time=-0.5 if phase == 0 else 0.0, side_x=15.0 if phase == 0 else None)
    pp = wall_state(n, 31, sys, vel=speed, omega=50.0)
    if speed < 100.0:   # twelve clumps on one spot: more near sphere pairs than a list holds
        pp["rr"][-12:] = pp["rr"][-12] + 0.02 * np.random.default_rng(3).random((12, 3))
        af3d.sphere_centres(pp)
    if nflumes > 1:
        sys, fun, pp = np.stack([sys] * nflumes), np.stack([fun] * nflumes), np.concatenate([pp] * nflumes)
    with start(af3d, sys, fun, pp, mode, phase, speed, nflumes) as kept, \
            start(af3d, sys, fun, pp, mode, phase, speed, nflumes) as new:
        contacts = []
        new.contact_count()
        for _ in range(STEPS):
            new.step(1)
            new.import_particles(*new.export_particles())
            contacts.append(new.contact_count())
        kept.contact_count()
        kept.step(STEPS)
        assert kept.contact_count() == sum(contacts) and sum(contacts) > 0
        for x, y in zip(kept.export_particles(), new.export_particles()):
            assert x.tobytes() == y.tobytes()
        if speed < 100.0:
            assert kept.list_overflows() > 0


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1.04, 1.06, 1.5])
def test_clumps_up_to_and_past_the_reach(af3d, mode, scale):
    """The largest clump of the flume's rmax, 5 % more (the largest the lists reach for) and more
    than that (every clump searches its cells): kept lists equal new ones, bit for bit."""
    from tests.states import flume_system, wall_state
    n = 301
    sys, fun = flume_system(n)
    pp = wall_state(n, 43, sys, vel=200.0, omega=50.0)
    pp["radius"][::7] = scale * float(np.ravel(sys["rmax"])[0])
    af3d.sphere_centres(pp)
    with start(af3d, sys, fun, pp, mode, 1, 200.0, 1) as kept, start(af3d, sys, fun, pp, mode, 1, 200.0, 1) as new:
        for _ in range(STEPS):
            new.step(1)
            new.import_particles(*new.export_particles())
        kept.step(STEPS)
        assert kept.contact_count() > 0
        for x, y in zip(kept.export_particles(), new.export_particles()):
            assert x.tobytes() == y.tobytes()
