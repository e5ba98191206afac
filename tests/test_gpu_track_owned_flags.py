"""The owned schedule's flag word at the counts where a field of it could be cut off or run over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import _lib, engine, workloads as W
from tests.test_gpu_track_f64_units import field, rk4, winding


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


@pytest.mark.parametrize("prec,scale", [("f64", s) for s in (1e3, 1e14, 1e18, 1e30, 1e40)] +
                         [("f32c", s) for s in (1e3, 1e14, 1e18, 1e30)])
@pytest.mark.parametrize("n_p", [3, 70])
def test_any_finite_field(prec, scale, n_p):
    """Fields from the counted range to 1e40 T, over one step that deflects by some 1e-3.  Bounds, of the
    deflection: FP64 a few 2^-53 of a velocity 1000 times as large, so 1e-12; FP32c 1e-5 (test_gpu_track_owned.py)."""
    kl, p0 = winding(5000)
    kl = kl * scale
    ps = W.single_dipole_particles(n_p, seed=1)
    ps[:, 3:6] = np.roll(ps[:, 3:6], 1, axis=1)          # across the field, which is along x
    length = float(1e-3 * ps[0, 8] * ps[0, 6] / (ps[0, 7] * np.linalg.norm(field(kl, p0, ps[:1, 0:3]))))
    out = engine.track(engine.DesignSet([(kl, p0, np.zeros((0, 16)))]), ps, length, length, prec)[0]
    _, v = rk4(ps, kl, p0, length, 1)
    turn = np.linalg.norm(v - ps[:, 3:6], axis=1)
    assert turn.min() > 1e-4 * np.linalg.norm(v[0])
    bound = 1e-12 if prec == "f64" else 1e-5
    assert (np.linalg.norm(out[:, 3:6] - v, axis=1) <= bound * turn).all()
