"""Accuracy of the FP64 field sums of tracks, against 80-bit sums.

One RK4 step with (e / m) B dt of some hundreds on protons that all but stand still: their velocity
becomes the step's fourth-order polynomial in the field, four times as sensitive to it.

Bound, of the 2-norm over the protons: a sub-block's sum of 32 terms is good to a few 2^-53 of its
field, the several hundred that matter add up at random, and the step rounds a few times: 2^-52.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import engine, workloads as W

LD = np.longdouble
POINTS = 24


def field(kl, p0, pts):
    out = np.zeros((len(pts), 3), LD)
    for i, p in enumerate(pts):
        r = p.astype(LD) - p0
        out[i] = (np.cross(kl.astype(LD), r) / np.sqrt((r * r).sum(1))[:, None] ** 3).sum(0)
    return out


def step(v, B, kq):
    f = lambda v: kq * np.cross(v, B)
    v = v.astype(LD)
    k1 = f(v)
    k2 = f(v + k1 / 2)
    k3 = f(v + k2 / 2)
    k4 = f(v + k3)
    return v + (k1 + 2 * k2 + 2 * k3 + k4) / 6


def design(part):
    rng = np.random.default_rng(part)
    if part is None:
        obj, pts = W.build_single_dipole()[1], W.field_map_points(POINTS, 3)
    else:
        obj = W.build_gantry_section(part_per_winding=part)
        s = rng.uniform(0.3, 0.9 * obj.get_length(), POINTS)
        pts = np.array([(obj.point_at(float(x)).x, obj.point_at(float(x)).y, 0.0) for x in s])
        pts += rng.uniform(-0.01, 0.01, pts.shape)
    return engine.host_design(engine.magnet_list(obj)), pts


@pytest.mark.parametrize("part", [None, 60, 120, 360], ids=["dipole", "60", "120", "360"])
def test_field_of_a_step(part):
    (kl, p0, _), pts = design(part)
    ds = engine.DesignSet([(kl, p0, np.zeros((0, 16)))])
    v = np.random.default_rng(1).normal(size=(POINTS, 3)) * 1e-28
    want = step(v, field(kl, p0, pts), LD(500.0))
    for n in (8, POINTS, 2048):                 # blocks of 8, of 32, and more blocks than there are SMs
        at = np.arange(n) % POINTS
        rec = np.zeros((n, 10))
        rec[:, 0:3], rec[:, 3:6] = pts[at], v[at]
        rec[:, 6], rec[:, 7], rec[:, 8] = 1.0, 500.0, 1.0
        out = engine.track(ds, rec, 1.0, 1.0, "f64")[0][:, 3:6]
        err = np.sqrt(((out.astype(LD) - want[at]) ** 2).sum() / (want[at] ** 2).sum()) / 4
        assert err <= 2.0 ** -52, (n, float(err))
