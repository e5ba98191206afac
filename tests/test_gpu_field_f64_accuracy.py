"""FP64 fields against 80-bit sums, from the bore to far outside where the terms cancel, and the same
bits for a point whatever its call looks like (from five points on).

Bound, of the 2-norm over a set's points: fields in hi + lo FP32 pairs are kept where their rounding is
below 3e-17 |B| sqrt(n / 256) (4e-16 of |B| in the dipole), others are FP64 sums of 32-segment sub-blocks, each good to 2^-52 of its sum of
|term|, adding up at random.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import QS, LocalCoordinateSystem, MM, P3, _lib, engine, workloads as W

LD = np.longdouble
NONE = np.zeros((0, 16))


def winding(n):
    """n segments of a tilted winding of radius 0.1 m, 120 a turn."""
    t = np.arange(n + 1) * (2 * np.pi / 120)
    w = np.stack([0.1 * np.cos(t), 0.1 * np.sin(t), 0.003 * t + 0.08 * np.sin(t)], 1)
    return 1e-7 * 9000.0 * (w[1:] - w[:-1]), 0.5 * (w[1:] + w[:-1])


def design(name):
    if name == "dipole":
        return engine.host_design(engine.magnet_list(W.build_single_dipole()[1]))[:2]
    if name == "section 60":
        return engine.host_design(engine.magnet_list(W.build_gantry_section(part_per_winding=60)))[:2]
    return winding(int(name))


def exact(kl, p0, pts):
    """(field, 2-norm over sub-blocks of their sum of |term|)"""
    B, mag = np.zeros((len(pts), 3), LD), np.zeros(len(pts))
    for i, p in enumerate(pts):
        r = p.astype(LD) - p0
        t = np.cross(kl.astype(LD), r) / np.sqrt((r * r).sum(1))[:, None] ** 3
        B[i] = t.sum(0)
        a = np.pad(np.sqrt((t * t).sum(1)).astype(float), (0, -len(t) % 32)).reshape(-1, 32).sum(1)
        mag[i] = np.sqrt((a * a).sum())
    return B, mag


@pytest.mark.parametrize("distance", [0.0, 0.3, 1.0, 5.0, 50.0, 500.0])
@pytest.mark.parametrize("name", ["2047", "2048", "5000", "dipole", "section 60"])
def test_error(name, distance):
    kl, p0 = design(name)
    rng = np.random.default_rng(int(distance * 10))
    at = p0[rng.integers(0, len(p0), 16)]
    if distance == 0.0:          # on the axis of a turn
        pts = np.array([p0[max(0, i - 60):i + 60].mean(0) for i in rng.integers(200, len(p0) - 200, 16)])
    else:
        u = rng.normal(size=(16, 3))
        pts = (at if distance < 1.0 else p0.mean(0)) + distance * u / np.linalg.norm(u, axis=1)[:, None]
    B, mag = exact(kl, p0, pts)
    size = np.sqrt((B * B).sum(1)).astype(float)
    for n in (8, 16):
        got = np.concatenate([engine.field_at_points(engine.DesignSet([(kl, p0, NONE)]), pts[i:i + n], "f64")
                              for i in range(0, 16, n)])
        err = np.sqrt(((got.astype(LD) - B) ** 2).sum(1)).astype(float)
        assert np.sqrt((err ** 2).sum()) <= np.sqrt(((4e-16 * size + 2.0 ** -52 * mag) ** 2).sum())


@pytest.mark.parametrize("name", ["1", "31", "513", "2049", "6000", "dipole"])
def test_same_bits_in_any_call(name):
    """Shapes of all kinds (entries of sub-blocks and of chunks, splits, narrow and wide CTAs, none), and with
    a workspace that is short or missing."""
    kl, p0 = design(name)
    qs = np.stack([engine.analytic_record(QS(LocalCoordinateSystem(P3(0, 0, 0), -P3.x_direct(), P3.y_direct()), 0.27, 5,
                                              20, 100 * MM))])
    ds = engine.DesignSet([(kl, p0, qs)])
    rng = np.random.default_rng(4)
    n = 5000
    pts = p0[rng.integers(0, len(p0), n)] * [0.5, 0.5, 1.0] + rng.uniform(-0.02, 0.02, (n, 3))
    pts[::7] += rng.uniform(-2.0, 2.0, pts[::7].shape)          # some outside, among the others
    want = engine.field_at_points(ds, pts, "f64")
    assert np.isfinite(want).all()
    for m in (5, 8, 9, 16, 17, 31, 33, 130, 352, 353, 1100):
        for a in (0, 1777):
            assert np.array_equal(engine.field_at_points(ds, pts[a:a + m], "f64"), want[a:a + m]), m
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    for m in (5, 40, 400, 5000):
        d = torch.from_numpy(pts[:m].copy()).cuda()
        full = lib.cct_field_work_bytes(len(kl), m, 0)
        for part in (0.0, 0.3, 1.0):
            work, out = torch.empty(max(int(full * part), 8), dtype=torch.uint8, device="cuda"), torch.empty_like(d)
            _lib.check(lib.cct_field_f64_ws(ds.kls.data_ptr(), ds.p0s.data_ptr(), len(kl), ds.qs.data_ptr(), 1,
                                            d.data_ptr(), m, out.data_ptr(), work.data_ptr() if part else 0,
                                            int(full * part), st), "field")
            assert np.array_equal(out.cpu().numpy(), want[:m]), (m, part)


def test_fields_over_their_points():
    """Fields written over the points they are of: all in FP64, as good as any."""
    kl, p0 = design("6000")
    ds = engine.DesignSet([(kl, p0, NONE)])
    rng = np.random.default_rng(4)
    for m in (3, 300, 1000):
        pts = p0[rng.integers(0, len(p0), m)] * [0.5, 0.5, 1.0]
        want = engine.field_at_points(ds, pts, "f64")
        d = torch.from_numpy(pts.copy()).cuda()
        _lib.check(_lib.load().cct_field_f64(ds.kls.data_ptr(), ds.p0s.data_ptr(), 6000, 0, 0, d.data_ptr(), m,
                                             d.data_ptr(), torch.cuda.current_stream().cuda_stream), "field")
        assert np.abs(d.cpu().numpy() - want).max() <= 1e-14 * np.abs(want).max()
