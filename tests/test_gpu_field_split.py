"""Field calls of every launch shape (a few points, narrow and wide CTAs, segment splits with
ragged ends) against a plain numpy FP64 sum.

Bounds: an FP64 sum of N <= 6000 terms is within N 2^-53 < 1e-12 of sum |term|, the moment form
multiplying that by |p - o| / |r| (<= 10 here); an FP32 sum over 128-segment tiles is within
128 2^-24 < 1e-5 of it (offsets, weights and the sum, each rounded to FP32).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import QS, LocalCoordinateSystem, MM, P3, _lib, engine

BOUND = {"f64": 1e-11, "f32c": 1e-5}
QS_AT = QS(LocalCoordinateSystem(P3(0, 0, 0), -P3.x_direct(), P3.y_direct()), 0.27, 5, 20, 100 * MM)


def winding(n, seed=3):
    """(kl, p0) of n segments of a solenoid of radius 0.1 m around z, 90 a turn, and one far turn."""
    t = np.arange(n + 1) * (2 * np.pi / 90)
    w = np.stack([0.1 * np.cos(t), 0.1 * np.sin(t), 0.001 * t], 1)
    w[n // 2:, 2] += 1.5                        # a jump inside a tile
    return 1e-7 * 9000.0 * (w[1:] - w[:-1]), 0.5 * (w[1:] + w[:-1])


def points(n, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(-0.04, 0.04, (n, 2)), rng.uniform(-0.1, 0.3, (n, 1))], 1)


def plain(kl, p0, qs, pts):
    r = pts[:, None, :] - p0[None]
    t = np.cross(kl[None], r) / np.linalg.norm(r, axis=2)[..., None] ** 3
    return t.sum(1), np.linalg.norm(t, axis=2).sum(1)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_seg", [1, 31, 33, 127, 128, 129, 257, 2049, 6000])
def test_launch_shapes(prec, n_seg):
    kl, p0 = winding(n_seg)
    none = np.zeros((0, 16))
    ds = engine.DesignSet([(kl[:1], p0[:1], none), (kl, p0, none)])       # not the set's first design
    for n in (1, 2, 3, 5, 8, 9, 31, 32, 33, 96, 97, 127, 129, 383, 385, 513):
        pts = points(n, n)
        want, mag = plain(kl, p0, none, pts)
        got = engine.field_at_points(ds, pts, prec, design=1)
        assert (np.linalg.norm(got - want, axis=1) <= BOUND[prec] * mag).all(), (n, n_seg)
        assert np.array_equal(engine.field_at_points(ds, pts, prec, design=1), got)   # a fixed order


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_analytic_magnets_and_no_workspace(prec):
    """The QS part is added once, after the splits; a caller without a workspace gets the same
    field to rounding."""
    kl, p0 = winding(3000)
    qs = np.stack([engine.analytic_record(QS_AT)])
    ds = engine.DesignSet([(kl, p0, qs)])
    bare = engine.DesignSet([(kl, p0, np.zeros((0, 16)))])
    zero = engine.DesignSet([(kl[:0], p0[:0], qs)])
    lib = _lib.load()
    for n in (1, 7, 40, 600):
        pts = points(n, 5)
        got = engine.field_at_points(ds, pts, prec)
        q = engine.field_at_points(zero, pts, prec)
        assert n < 600 or np.abs(q).max() > 0      # a quarter of the points lie inside the magnet
        _, mag = plain(kl, p0, qs, pts)
        parts = engine.field_at_points(bare, pts, prec) + q
        assert (np.abs(got - parts).max(1) <= 1e-15 * (mag + 1.0)).all()
        d_pts, out = torch.from_numpy(pts).cuda(), torch.empty((n, 3), dtype=torch.float64, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        if prec == "f64":
            rc = lib.cct_field_f64(ds.kls.data_ptr(), ds.p0s.data_ptr(), 3000, ds.qs.data_ptr(), 1, d_pts.data_ptr(),
                                   n, out.data_ptr(), st)
        else:
            rc = lib.cct_field_f32c(ds.packed().data_ptr(), 0, ds.qs.data_ptr(), 1, d_pts.data_ptr(), n,
                                    out.data_ptr(), st)
        _lib.check(rc, "field without workspace")
        assert (np.abs(out.cpu().numpy() - got).max(1) <= BOUND[prec] * mag).all()
