"""The FP64 field sum on the FP32 pipe (hi + lo pairs) and its hand-overs to plain FP64, against an
extended-precision sum.

Bound: the rounding of one pair term is below 2^-43 of it (|r| 2^-47, |r|^2 and the correction of
the reciprocal root ten roundings of 2^-48 each, times 3/2), so the sum is within 1.2e-13 of
sum |term| whatever the points and currents; plain FP64 is far inside that.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import engine

BOUND = 1.2e-13
N_SEG = 2500            # 78 sub-blocks of 32, a ragged one of 4; at least 2048 segments


def winding(n):
    t = np.arange(n + 1) * (2 * np.pi / 90)
    w = np.stack([0.1 * np.cos(t), 0.1 * np.sin(t), 0.001 * t], 1)
    return 1e-7 * 9000.0 * (w[1:] - w[:-1]), 0.5 * (w[1:] + w[:-1])


def wide_sum(kl, p0, pts):
    out, mag = np.zeros((len(pts), 3), np.longdouble), np.zeros(len(pts))
    for i, p in enumerate(pts):
        r = p.astype(np.longdouble) - p0
        t = np.cross(kl.astype(np.longdouble), r) / np.sqrt((r * r).sum(1))[:, None] ** 3
        out[i], mag[i] = t.sum(0), np.sqrt((t * t).sum(1)).sum()
    return out, mag


def points(p0, n):
    """Inside the bore, close to segments, in the bore's surroundings, and far away."""
    rng = np.random.default_rng(n)
    pts = rng.uniform(-0.06, 0.06, (n, 3)) + [0.0, 0.0, 0.05]
    near = rng.integers(0, len(p0), n // 4)
    pts[:n // 4] = p0[near] * [0.99, 0.99, 1.0]              # 1 mm from a segment (7 mm apart)
    pts[n // 4:n // 4 + 2] = p0[near[:2]] * [0.72, 0.72, 1.0]    # at 28 mm, the limit of "near"
    pts[-1], pts[-2], pts[-3] = [3.0e4, 1.0, -2.0], [0.0, -9.99e3, 10.0], [2.0e7, 0.0, 3.0e5]
    return pts


@pytest.mark.parametrize("n", [24, 60, 200])
@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e-20, 1e25, 0.0])
def test_sum_and_hand_overs(n, scale):
    kl, p0 = winding(N_SEG)
    pts = points(p0, n)
    ds = engine.DesignSet([(kl * scale, p0, np.zeros((0, 16)))])
    got = engine.field_at_points(ds, pts, "f64")
    want, mag = wide_sum(kl, p0, pts)
    err = np.sqrt(((got.astype(np.longdouble) - want * scale) ** 2).sum(1))
    assert (err <= BOUND * mag * scale).all(), (err / np.maximum(mag * scale, 1e-300)).max()
    perm = np.random.default_rng(0).permutation(n)      # a point's field does not depend on its neighbours
    assert np.array_equal(engine.field_at_points(ds, pts[perm], "f64"), got[perm])


def test_mixed_and_nonfinite():
    kl, p0 = winding(N_SEG)
    kl[100:200] = 0.0
    kl[300:364] *= 1e-22                                 # below the range of one sub-block, among others
    pts = points(p0, 64)
    ds = engine.DesignSet([(kl, p0, np.zeros((0, 16)))])
    got = engine.field_at_points(ds, pts, "f64")
    want, mag = wide_sum(kl, p0, pts)
    assert (np.sqrt(((got.astype(np.longdouble) - want) ** 2).sum(1)) <= BOUND * mag).all()
    bad = pts.copy()
    bad[5, 1] = np.nan
    out = engine.field_at_points(ds, bad, "f64")
    keep = np.arange(64) != 5
    assert np.isnan(out[5]).all() and np.array_equal(out[keep], got[keep])
    kl[7, 2] = np.inf
    assert not np.isfinite(engine.field_at_points(engine.DesignSet([(kl, p0, np.zeros((0, 16)))]), pts, "f64")).all(1).any()
