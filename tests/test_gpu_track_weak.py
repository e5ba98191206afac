"""FP32c tracks through weak magnets: FP32 arithmetic is the same whatever power of two the currents are
scaled by, so the track through a design at 2^-25 of its currents, of protons with 2^25 times the charge,
is the first one's as far as the sums between warps and CTAs hold their bits.

Bound: fields of about 1 T at 2^-25 are 3e-8 T; some 2000 sums rounded at 2^-54 T, at random, are 7e-16 T,
2e-8 of that, 5e-8 at most of the points; one RK4 step is four times as sensitive.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import engine, workloads as W


@pytest.mark.parametrize("n_p", [65, 100, 256, 700])
def test_weak_currents(n_p):
    kl, p0, _ = engine.host_design(engine.magnet_list(W.build_single_dipole()[1]))
    rec = np.zeros((n_p, 10))
    rec[:, 0:3] = W.field_map_points(n_p, 5)
    rec[:, 3:6] = np.random.default_rng(1).normal(size=(n_p, 3)) * 1e-28
    rec[:, 6], rec[:, 7], rec[:, 8] = 1.0, 500.0, 1.0
    out = []
    for scale in (1.0, 2.0 ** -25):
        rec[:, 7] = 500.0 / scale
        ds = engine.DesignSet([(kl * scale, p0, np.zeros((0, 16)))])
        out.append(engine.track(ds, rec, 1.0, 1.0, "f32c")[0][:, 3:6])
    err = np.linalg.norm(out[1] - out[0], axis=1) / np.linalg.norm(out[0], axis=1)
    assert np.sqrt((err ** 2).mean()) <= 4 * 5e-8
