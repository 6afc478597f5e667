"""The force pass at small counts (csrc/af3d_wide.cuh, up to 20,480 clumps in a context) against
the pass for larger ones: one flume alone equals, bit for bit, the same flume twice in a context
that is past the limit, in both FP64 modes; and on both sides of the limit an exact step equals
the routines called one by one.  Bit equality: both passes add the same terms in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 20480


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


def state(n):
    from tests.states import flume_system, wall_state
    sys, fun = flume_system(n)
    return sys, fun, wall_state(n, 17, sys, vel=40.0, omega=50.0)


def started(af3d, sys, fun, pp, mode):
    e = af3d.Engine(sys, fun, ntags=0, fp_mode=mode)
    e.import_particles(pp)
    e.forces()
    e.swap_accel()
    e.step(1)   # past the re-grid that follows a run's first step
    return e


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [LIMIT // 2 + 1, LIMIT])
def test_both_passes_agree(af3d, mode, n):
    sys, fun, pp = state(n)
    with started(af3d, sys, fun, pp, mode) as one, \
            started(af3d, np.stack([sys] * 2), np.stack([fun] * 2), np.concatenate([pp] * 2), mode) as two:
        one.step(3)
        two.step(3)
        assert one.contact_count() > 0
        for x, y in zip(one.export_particles(), two.export_particles()):
            assert y[:n].tobytes() == x.tobytes() and y[n:].tobytes() == x.tobytes()


@pytest.mark.parametrize("n", [31, 33, LIMIT, LIMIT + 1])
def test_step_equals_routines(af3d, n):
    sys, fun, pp = state(n)
    with started(af3d, sys, fun, pp, 0) as step, started(af3d, sys, fun, pp, 0) as loop:
        step.step(2)
        for _ in range(2):
            loop.init_verlet()
            loop.advance_time()
            loop.rotate_vectors()
            loop.clear_forces()
            loop.cell_build()
            for nw in range(3):
                loop.force_hop(nw)
            loop.force_funnel()
            loop.force_fcorners()
            loop.force_walls()
            loop.force_part(0)
            loop.force_flume()
            loop.get_accel()
            loop.finish_verlet()
            loop.swap_accel()
        for x, y in zip(step.export_particles(), loop.export_particles()):
            assert x.tobytes() == y.tobytes()
