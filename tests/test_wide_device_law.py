"""The small-count force pass (csrc/af3d_wide.cuh) in fast mode under the device friction law, whose
rotation takes the FP64 formulas and whose limit is one wave of blocks: one flume alone equals, bit for bit,
the same flume twice in a context past the limit."""
import numpy as np
import pytest

from tests.test_wide import state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fast", "exact"])
@pytest.mark.parametrize("n", [10241, 19456, 19457])
def test_both_passes_agree_under_the_device_law(mode, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import avalancheflume3d_gb300 as af3d
    sys, fun, pp = state(n)

    def run(sys, fun, pp):
        with af3d.Engine(sys, fun, ntags=0, friction=af3d.FRICTION_DEV,
                         fp_mode=af3d.FP_FAST if mode == "fast" else af3d.FP_EXACT) as e:
            e.import_particles(pp)
            e.forces()
            e.swap_accel()
            e.step(4)
            return e.export_particles(), e.contact_count()

    one, contacts = run(sys, fun, pp)
    two, _ = run(np.stack([sys] * 2), np.stack([fun] * 2), np.concatenate([pp] * 2))
    assert contacts > 0
    for x, y in zip(one, two):
        assert y[:n].tobytes() == x.tobytes() and y[-n:].tobytes() == x.tobytes()
