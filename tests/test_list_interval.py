"""The interval of the near lists follows the flow (list_interval, csrc/af3d_internal.h): a flow that would
outrun the lists of 16 steps has them built every 8, 4 or 2 steps, and 16 again when it is slow;
the results are those of new lists in every step, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


def moving(pp, sys, speed):
    """The bed pp carried downslope at `speed`, its clumps with velocities of their own."""
    pp = pp.copy()
    pp["vv"] = 4.0 * np.random.default_rng(2).standard_normal((len(pp), 3))
    pp["vv"][:, 0] += speed * float(sys["cost"])
    pp["vv"][:, 2] -= speed * float(sys["sint"])
    return pp


def launches(af3d, e):
    import ctypes as C
    v = C.c_long()
    e._call("af3d_kernel_launches", C.byref(v))
    return v.value


@pytest.mark.parametrize("n,mode", [(1203, 0), (1203, 1), (21001, 1)])
def test_the_interval_follows_the_flow(af3d, n, mode):
    from avalancheflume3d_gb300.workloads import flume_2k, flume_state
    sys, fun, pp0 = flume_state(flume_2k(n=n, width=4.0, Lflume=80.0, layout="bed", overlap=2.0e-5))
    per_step = {}
    with af3d.Engine(sys, fun, ntags=0, fp_mode=mode) as e, af3d.Engine(sys, fun, ntags=0, fp_mode=mode) as new:
        for c in (e, new):
            c.import_particles(moving(pp0, sys, 0.0))
            c.step(1)   # past the first re-grid
        for speed in (100.0, 1300.0, 3000.0, 6000.0, 100.0):
            pp = moving(pp0, sys, speed)
            for c in (e, new):
                c.import_particles(pp)
                c.forces()   # whose lists tell the speed
                c.swap_accel()
            before = launches(af3d, e)
            e.step(16)
            per_step[speed] = launches(af3d, e) - before
            for _ in range(16):
                new.step(1)
                new.import_particles(*new.export_particles())
            for x, y in zip(e.export_particles(), new.export_particles()):
                assert x.tobytes() == y.tobytes(), speed
    # four launches (sort, lists) for each build after the first
    assert [per_step[v] - per_step[100.0] for v in (1300.0, 3000.0, 6000.0)] == [4, 12, 28], per_step
