"""A clump that outruns its near list (csrc/af3d_near.cu) or is not finite costs the clumps around it
alone: the others keep their lists and their results, bit for bit, whatever flume it is in, and a call
with it takes about as long as one without."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 40


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


def state(af3d, n, flumes=1):
    from avalancheflume3d_gb300.workloads import flume_2k, flume_state
    sys, fun, pp = flume_state(flume_2k(n=n, width=4.0 if n < 50000 else 20.0,
                                        Lflume=80.0 if n < 50000 else 200.0, layout="bed", overlap=2.0e-5))
    pp["vv"] += 4.0 * np.random.default_rng(2).standard_normal((n, 3))
    if flumes > 1:
        return np.stack([sys] * flumes), np.stack([fun] * flumes), np.concatenate([pp] * flumes)
    return sys, fun, pp


def steps(af3d, sys, fun, pp, one_by_one=False):
    """(particles, accelerations, contacts, seconds, status) after STEPS steps past the first re-grid;
    one_by_one: every step from an import, so with lists of its own."""
    with af3d.Engine(sys, fun, ntags=0, fp_mode=af3d.FP_FAST) as e:
        still = pp.copy()
        still["vv"] = still["ww"] = 0.0
        e.import_particles(still)
        e.step(1)
        e.import_particles(pp)
        e.status()
        e.contact_count()
        t = time.perf_counter()
        status = 0
        for _ in range(STEPS if one_by_one else 1):
            try:
                e.step(1 if one_by_one else STEPS)
            except Exception:
                pass
            status |= e.status()
            if one_by_one:
                e.import_particles(*e.export_particles())
        t = time.perf_counter() - t
        return (*e.export_particles(), e.contact_count(), t, status)


@pytest.mark.parametrize("n,flumes", [(1201, 1), (24001, 1), (1201, 3)])
def test_a_runaway_through_the_bed(af3d, n, flumes):
    """One clump (of the last flume) shot along the bed, several cells a step: as with new lists a step."""
    sys, fun, pp = state(af3d, n, flumes)
    pp["vv"][-n // 2] = (-3.0e5, 1.0e3, 0.0)
    kept, new = steps(af3d, sys, fun, pp), steps(af3d, sys, fun, pp, True)
    assert kept[3] > 0
    for x, y in zip(kept[:4], new[:4]):
        assert np.asarray(x).tobytes() == np.asarray(y).tobytes()


@pytest.mark.parametrize("n", [1201, 24001])
def test_a_clump_that_is_not_finite(af3d, n):
    """A clump whose spin is NaN: the clumps it cannot meet (all others) as with new lists a step."""
    sys, fun, pp = state(af3d, n)
    pp["ww"][n // 3] = np.nan
    kept, new = steps(af3d, sys, fun, pp), steps(af3d, sys, fun, pp, True)
    for x, y in zip(kept[:4], new[:4]):
        assert np.asarray(x).tobytes() == np.asarray(y).tobytes()


@pytest.mark.parametrize("what", ["runaway", "nan"])
def test_the_others_keep_their_pace(af3d, what):
    """100,003 clumps, one of them fast or not finite: far from a search of every clump by every
    other, which would take minutes."""
    sys, fun, pp = state(af3d, 100003)
    plain = steps(af3d, sys, fun, pp)[4]
    if what == "nan":
        pp["ww"][50000] = np.nan
    else:
        pp["vv"][50000] = (-3.0e5, 1.0e3, 0.0)
    assert steps(af3d, sys, fun, pp)[4] < 10.0 * plain + 0.1
