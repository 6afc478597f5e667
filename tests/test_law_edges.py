"""The contact law where its shortcuts must not be taken: a negative friction puts a contact whose
displacement the gate cuts into the Coulomb branch (|0| > mu N, force_part.cu:224-232), and a time step of
zero makes the displacement's rate 0 / 0.  One force pass of moving, overlapping clumps against the oracle,
bit for bit."""
import numpy as np
import pytest

from oracle.pyoracle import FRICTION_DEV, FRICTION_HST, OracleRun, dense_state
from tests.states import flume_system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def af3d():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    af3d.lib()
    return af3d


@pytest.mark.parametrize("friction", [FRICTION_HST, FRICTION_DEV])
@pytest.mark.parametrize("n", [400, 21000])   # either shape of the force pass
@pytest.mark.parametrize("mu,dt", [(-0.3, 2e-6), (0.0, 2e-6), (0.5, 0.0)])
def test_force_pass_equals_the_oracle(af3d, oracle, friction, n, mu, dt):
    sys, fun = flume_system(n, time=0.001)
    sys["mu_pp"] = mu
    sys["fr_fact_pp"] = mu / 1.0e12
    sys["dt"], sys["hdt"] = dt, 0.5 * dt
    pp = dense_state(n, 3, sys, box=(1.0, 8.0, 26.0) if n < 1000 else (8.0, 8.0, 26.0))
    run = OracleRun(oracle, sys, fun, pp)
    assert run.forces(1, friction) == 0
    with af3d.Engine(sys, fun, ntags=0, friction=friction) as e:
        e.set_grid(run.cp)
        e.import_particles(pp)
        try:
            e.forces()
        except Exception:
            assert dt == 0.0   # NaN accelerations are raised
        F, T = e.get_forces()
        assert e.contact_count() > n // 8
        for got, want in ((F, run.bufs["F"]), (T, run.bufs["T"])):
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.where(nan, 0.0, got).tobytes() == np.where(nan, 0.0, want).tobytes()
