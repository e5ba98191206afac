"""The dataflow and grid-barrier schedules on inputs that do take them (cct_test_plan_schedule): results
against RK4 in numpy FP64, and their bounded waits.

Bounds as in test_gpu_track_owned.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import _lib, engine, workloads as W
from cctpy_gb300.adjoint import segment_gradient
from tests.test_gpu_track_f64_units import winding
from tests.test_gpu_track_owned import NONE, check

OWNED, DATAFLOW, BARRIERS = 0, 1, 2
PREC = {"f64": 0, "f32c": 1}
FRAME = np.array([0.9, 0.02, 0.0, 0.6, 0.8, 0.0, 0.0, 0.0, 1.0])


def schedule(ds, n_p, prec, scratch):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return _lib.load().cct_test_plan_schedule(ds.h_seg_off.ctypes.data, ds.n_designs, n_p, PREC[prec], sms, 3 * sms, scratch)


def little_scratch(ds, n_p, prec):
    """The most scratch that the owned schedule's accumulators do not fit in."""
    fits = [s for s in range(256, 1 << 18, 256) if schedule(ds, n_p, prec, s) == BARRIERS]
    assert fits and schedule(ds, n_p, prec, 1 << 40) == OWNED
    return fits[-1]


def track(ds, ps, length, step, prec, scratch):
    p = torch.from_numpy(np.tile(ps, (ds.n_designs, 1, 1))).cuda()
    buf = torch.empty(scratch + 256, dtype=torch.uint8, device="cuda")
    rc = _lib.load().cct_track(ds.kls.data_ptr(), ds.p0s.data_ptr(), ds.seg_off.data_ptr(),
                               ds.packed().data_ptr() if prec == "f32c" else 0, 0, ds.qs_off.data_ptr(), ds.n_designs,
                               p.data_ptr(), len(ps), length, step, PREC[prec], buf.data_ptr() + (-buf.data_ptr()) % 256,
                               scratch, torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "cct_track")
    return p.cpu().numpy()


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [4, 8, 16, 17, 33, 70])
def test_grid_barriers(prec, n_p):
    kl, p0 = winding(4001)
    ds = engine.DesignSet([(kl, p0, NONE)])
    ps = W.single_dipole_particles(n_p, seed=n_p)
    out = track(ds, ps, 0.0295, 0.01, prec, little_scratch(ds, n_p, prec))
    check(out[0], ps, kl, p0, 0.0295, 3, prec)


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n_p", [1, 9, 16, 17, 40])
def test_dataflow(prec, n_p):
    designs = [(*winding(n), NONE) for n in (600, 1, 131)]
    ds = engine.DesignSet(designs * 54)                 # 162 designs: more blocks than SMs
    ps = W.single_dipole_particles(n_p, seed=n_p)
    assert schedule(ds, n_p, prec, 1 << 40) == DATAFLOW
    out = engine.track(ds, ps, 0.0295, 0.01, prec)
    for d, (kl, p0, _) in enumerate(designs):
        check(out[d], ps, kl, p0, 0.0295, 3, prec)
        assert (out[d::3] == out[d]).all()


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_dataflow_wait_runs_out(prec):
    ds = engine.DesignSet([(*winding(600), NONE)] * 160)
    ps = W.single_dipole_particles(2, seed=1)
    assert schedule(ds, 2, prec, 1 << 40) == DATAFLOW
    lib = _lib.load()
    lib.cct_test_set_flow_fault(1, 300)
    try:
        with pytest.raises(_lib.CctTimeoutError):
            engine.track(ds, ps, 0.0295, 0.01, prec)
    finally:
        lib.cct_test_set_flow_fault(0, 0)
    assert np.isfinite(engine.track(ds, ps, 0.0295, 0.01, prec)).all()


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_grid_barrier_wait_runs_out(prec):
    ds = engine.DesignSet([(*winding(4000), NONE)])
    ps = W.single_dipole_particles(16, seed=1)
    scratch = little_scratch(ds, 16, prec)
    lib = _lib.load()
    lib.cct_test_set_barrier_fault(1, 300)
    try:
        with pytest.raises(_lib.CctTimeoutError):
            track(ds, ps, 0.0295, 0.01, prec, scratch)
        with pytest.raises(_lib.CctTimeoutError):          # (its state and its reverse sweep)
            segment_gradient(ds, ps, 0.0295, 0.01, FRAME[None], precision=prec)
    finally:
        lib.cct_test_set_barrier_fault(0, 0)
    assert np.isfinite(track(ds, ps, 0.0295, 0.01, prec, scratch)).all()
