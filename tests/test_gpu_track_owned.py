"""The owned schedule (a share of a particle block's segments on every SM, counted fixed-point
accumulators) over its block sizes, designs, shares that do not fit in shared memory or hold several
units, fields beyond the counted range and QS magnets, against RK4 in numpy FP64.

Bounds: FP64 as in test_gpu_track_f64_units.py; FP32c fields are within 1e-5 of sum |term|
(test_gpu_field_split.py), so after a deflection below 0.1 rad velocities are within 1e-6 of |v| and
positions over 30 mm within 3e-8 m.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import MM, P3, QS, LocalCoordinateSystem, engine, workloads as W
from tests.test_gpu_track_f64_units import field, rk4, winding

NONE = np.zeros((0, 16))
VEL = {"f64": 2e-14, "f32c": 1e-6}
POS = {"f64": 1e-14, "f32c": 3e-8}


def check(out, ps, kl, p0, length, steps, prec, vel=None):
    p, v = rk4(ps, kl, p0, length, steps)
    assert np.abs(out[:, 0:3] - p).max() <= (POS[prec] if vel is None else vel * length)
    assert np.abs(out[:, 3:6] - v).max() <= (vel or VEL[prec]) * np.abs(v).max()
    assert np.array_equal(out[:, 6:9], ps[:, 6:9]) and np.allclose(out[:, 9], ps[:, 9] + length, atol=1e-15)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [1, 8, 9, 15, 16, 17, 32, 33, 64])
def test_blocks_and_designs(prec, n_p):
    ps = W.single_dipole_particles(n_p, seed=n_p)
    for sizes in ([4000], [0], [1, 130, 5001][:max(1, 64 // n_p)]):
        designs = [(*winding(s), NONE) for s in sizes]
        out = engine.track(engine.DesignSet(designs), ps, 0.0295, 0.01, prec)
        for d, (kl, p0, _) in enumerate(designs):
            check(out[d], ps, kl, p0, 0.0295, 3, prec)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [3, 20])
def test_chunks_beyond_shared_memory(prec, n_p):
    """Two designs of 400 000 segments: about 42 tiles or 165 sub-blocks a CTA, of which 36 and 75 fit."""
    kl, p0 = winding(5000)
    kl, p0 = np.tile(kl, (80, 1)) / 80, np.tile(p0, (80, 1))
    ps = W.single_dipole_particles(n_p, seed=n_p)
    half = engine.DesignSet([(kl, p0, NONE), (kl * 0.5, p0, NONE)])
    out = engine.track(half, ps, 0.0195, 0.01, prec)
    for d, f in enumerate((1.0, 0.5)):
        check(out[d], ps, kl[:5000] * 80 * f, p0[:5000], 0.0195, 2, prec)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [65, 100, 130, 257, 600])
def test_larger_blocks(prec, n_p):
    """Blocks of 128 and 256 (FP32c; two protons a lane, quads split by particle sub-block) and several
    blocks a design, the last ragged."""
    kl, p0 = winding(4000)
    ps = W.single_dipole_particles(n_p, seed=n_p)
    out = engine.track(engine.DesignSet([(kl, p0, NONE)]), ps, 0.0295, 0.01, prec)[0]
    check(out, ps, kl, p0, 0.0295, 3, prec)


@pytest.mark.parametrize("n_designs,n_p", [(5, 16), (1, 70), (2, 33)])
def test_several_streamed_units(n_designs, n_p):
    """FP32c shares of several units past shared memory, with units of 43 tiles (an odd number: the
    half-warp blocks' pairs of warps change their ring slots at every unit) and of 32."""
    kl, p0 = winding(5000)
    kl, p0 = np.tile(kl, (200, 1)) / 200, np.tile(p0, (200, 1))
    ps = W.single_dipole_particles(n_p, seed=n_p)
    ds = engine.DesignSet([(kl * (1.0 + 0.1 * d), p0, NONE) for d in range(n_designs)])
    try:
        for units in (2, 0):
            engine.set_units_per_cta(units)
            out = engine.track(ds, ps, 0.0195, 0.01, "f32c")
            for d in range(n_designs):
                check(out[d], ps, kl[:5000] * 200 * (1.0 + 0.1 * d), p0[:5000], 0.0195, 2, "f32c")
    finally:
        engine.set_units_per_cta(0)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_unit_fields_beyond_the_counted_range(prec):
    """A proton starting 0.2 mm from a segment (48 T): the other protons' tracks are those of a batch
    without it, bit for bit."""
    kl, p0 = winding(5000)
    ps = W.single_dipole_particles(4, seed=1)
    ps[2, 0:3] = p0[2200] + [0.0, 0.0, 2e-4]
    ds = engine.DesignSet([(kl, p0, NONE)])
    out = engine.track(ds, ps, 1.95e-4, 1e-4, prec)[0]
    assert np.abs(field(kl, p0, ps[2:3, 0:3])).max() > 40
    check(out, ps, kl, p0, 1.95e-4, 2, prec, vel=1e-12 if prec == "f64" else 1e-4)
    keep = [0, 1, 3]
    assert np.array_equal(engine.track(ds, ps[keep], 1.95e-4, 1e-4, prec)[0], out[keep])


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [4, 70])
@pytest.mark.parametrize("off", [1e-3, 1e-4, 1e-5, 2e-6])
def test_fields_beyond_fixed_point(prec, n_p, off):
    """Protons 1 mm to 2 um from a segment (6 T to 1.5 MT: the uncounted words, the FP64 ones, FP32c also
    unconverted sums), deflected by 5e-6 to 3e-3 rad, next to others whose tracks do not change.  Bounds, of the
    deflection: FP64 the rounding of the distance, 1e-16 m, and of the sums; FP32c that of a local
    coordinate of 0.2 m, 1.2e-8 m, in 1 / r^2, and the usual 1e-5."""
    kl, p0 = winding(5000)
    ps = W.single_dipole_particles(n_p, seed=1)
    for j, s in ((2, 2200), (3, 4100)):
        ps[j, 0:3] = p0[s] + [off, 0.0, 0.0]
    ds = engine.DesignSet([(kl, p0, NONE)])
    length = 2e-3 * off
    out = engine.track(ds, ps, length, length / 1.95, prec)[0]
    near, keep = [2, 3], [j for j in range(n_p) if j not in (2, 3)]
    _, v = rk4(ps[near], kl, p0, length, 2)
    turn = np.linalg.norm(v - ps[near, 3:6], axis=1)
    assert turn.min() > 1e-6 * np.linalg.norm(v)
    bound = 1e-9 if prec == "f64" else 3e-8 / off + 1e-5
    assert (np.linalg.norm(out[near, 3:6] - v, axis=1) <= bound * turn).all()
    assert np.array_equal(engine.track(ds, ps[keep], length, length / 1.95, prec)[0], out[keep])


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_qs_edges_match_the_dataflow_schedule(prec):
    """Protons inside, outside and crossing the ends of a QS: the same in batches of 20 as in one of 65
    in 160 designs (the dataflow schedule, which tests every record at every stage)."""
    kl, p0 = winding(4000)
    qs = [QS(LocalCoordinateSystem(P3(x, 0, 0), P3.y_direct(), P3.z_direct()), 0.05, 5, 20, 100 * MM)
          for x in (0.02, 0.12, 0.5)]
    one = (kl, p0, np.stack([engine.analytic_record(q) for q in qs]))
    ds = engine.DesignSet([one])
    ps = W.single_dipole_particles(65, seed=3)
    ps[:, 0] += np.linspace(-0.11, 0.1, 65)
    many = engine.track(engine.DesignSet([one] * 160), ps, 0.0295, 0.003, prec)[0]
    few = np.concatenate([engine.track(ds, ps[i:i + 20], 0.0295, 0.003, prec)[0] for i in range(0, 65, 20)])
    assert np.abs(many[:, 0:3] - few[:, 0:3]).max() <= POS[prec]
    assert np.abs(many[:, 3:6] - few[:, 3:6]).max() <= VEL[prec] * np.abs(many[:, 3:6]).max()


@pytest.mark.parametrize("n_p", [1, 2, 3, 5, 7, 11])
def test_pieces_of_sub_blocks(n_p):
    """FP64 shares of a few sub-blocks, taken in pieces by lane groups of n_p; a proton 1 mm from the
    winding, so that single pieces fall back to plain FP64 (a deflection of 1e-5 rad)."""
    ps = W.single_dipole_particles(n_p, seed=n_p)
    near = ps.copy()
    for s in (2049, 9000, 20001):
        kl, p0 = winding(s)
        near[0, 0:3] = p0[s // 2] * [1.0, 1.01, 1.01]
        for rec, length, step in ((ps, 0.0295, 0.01), (near, 1e-4, 4e-5)):
            out = engine.track(engine.DesignSet([(kl, p0, NONE)]), rec, length, step, "f64")
            check(out[0], rec, kl, p0, length, 3, "f64")
