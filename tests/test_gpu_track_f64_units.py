"""FP64 tracking units (32-segment sub-blocks staged a warp at a time) at their edges: designs of
no, one, ragged and whole sub-blocks on both sides of the 2048-segment hand-over to plain FP64,
blocks of 16 and 32 with ragged last ones, every schedule, against RK4 in numpy FP64.

Bound: a pair term is within 1.2e-13 (test_gpu_field_df.py), so velocities after a deflection
below 0.1 rad are within 2e-14 of |v| (positions, over 30 mm, far closer) plus FP64 rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import engine, workloads as W

SIZES = [0, 1, 31, 33, 2047, 2048, 2111, 5000]


def winding(n):
    t = np.arange(n + 1) * (2 * np.pi / 90)
    w = np.stack([0.1 + 0.001 * t, 0.1 * np.cos(t), 0.1 * np.sin(t)], 1)     # around the x axis
    return 1e-7 * 9000.0 * (w[1:] - w[:-1]), 0.5 * (w[1:] + w[:-1])


def field(kl, p0, p):
    r = p[:, None] - p0[None]
    return (np.cross(kl[None], r) / np.linalg.norm(r, axis=2)[..., None] ** 3).sum(1)


def rk4(ps, kl, p0, length, steps):
    p, v, kq, sp = ps[:, 0:3], ps[:, 3:6], (ps[:, 7] / ps[:, 6])[:, None], ps[:, 8:9]
    h = length / sp / steps
    f = lambda p, v: (v, kq * np.cross(v, field(kl, p0, p)))
    for _ in range(steps):
        a1, b1 = f(p, v)
        a2, b2 = f(p + h / 2 * a1, v + h / 2 * b1)
        a3, b3 = f(p + h / 2 * a2, v + h / 2 * b2)
        a4, b4 = f(p + h * a3, v + h * b3)
        p, v = p + h / 6 * (a1 + 2 * a2 + 2 * a3 + a4), v + h / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
    return p, v


@pytest.mark.parametrize("n_p", [1, 16, 17, 33])
@pytest.mark.parametrize("sizes", [[s] for s in SIZES] + [SIZES + [2500]], ids=lambda s: "-".join(map(str, s)))
def test_units_match_numpy(sizes, n_p):
    none = np.zeros((0, 16))
    designs = [(*winding(s), none) for s in sizes]
    ds = engine.DesignSet(designs)
    ps = W.single_dipole_particles(n_p, seed=n_p)
    length, steps = 0.0295, 3
    out = engine.track(ds, ps, length, 0.01, "f64")
    for d, (kl, p0, _) in enumerate(designs):
        p, v = rk4(ps, kl, p0, length, steps)
        assert np.abs(out[d, :, 0:3] - p).max() <= 1e-14
        assert np.abs(out[d, :, 3:6] - v).max() <= 2e-14 * np.abs(v).max()
        assert np.array_equal(out[d, :, 6:9], ps[:, 6:9])
