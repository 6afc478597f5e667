"""The fast FP64 mode under the device friction law computes the same bits as it did when
tests/runs/fast_device.npz was written: under that law a last-bit difference anywhere in a step grows
by the ratio of speed to slip at every sliding pair, so a run shows whatever a kernel rounds
otherwise (af3d_physics.cuh)."""
import numpy as np
import pytest

from tests.runs.make_fast_device import PATH, RUNS, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", RUNS)
def test_fast_device_law_keeps_its_bits(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    with np.load(PATH) as want:
        for field, got in run(name).items():
            w = want["%s_%s" % (name, field)]
            assert got.tobytes() == w.tobytes(), (field, np.abs(got - w).max())
