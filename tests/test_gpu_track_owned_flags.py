"""The owned schedule's flag word at the counts where a field of it could be cut off or run over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import _lib, engine, workloads as W
from tests.test_gpu_track_f64_units import winding


@pytest.mark.parametrize("shares", [1, 2, 64, 85, 127, 128, 150])
def test_every_count_of_fields_that_are_not_finite(shares):
    """One current that is not finite in each of a number of CTAs' shares (a sub-block a CTA), on two of the
    field's components: the track ends in CCT_ERR_NONFINITE whatever the count, 256 among them."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if shares > sms:
        pytest.skip("fewer SMs than shares")
    kl, p0 = winding(32 * sms)
    kl[0:32 * shares:32] = [np.inf, 0.0, 0.0]
    ps = W.single_dipole_particles(1, seed=1)
    ds = engine.DesignSet([(kl, p0, np.zeros((0, 16)))])
    with pytest.raises(_lib.CctNonFiniteError):
        engine.track(ds, ps, 0.0095, 0.01, "f64")
