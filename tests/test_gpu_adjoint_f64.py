"""FP64 adjoint sums (separate kernels up to some 8000 segments, one pass from there on) at the edges
of their blocks, tiles and chunks, against torch autograd of the same RK4 track on the CPU.

Bound: both sides sum the same FP64 terms in other orders.  A field or a gradient here is a sum of N
terms that cancels by less than 100; a term is good to a few 2^-53, so a sum is within
100 (4 + sqrt(N)) 2^-53 < 1e-12 of itself, and the gradient's norm within some sums of that: 1e-11.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import engine, workloads as W
from cctpy_gb300.adjoint import segment_gradient
from tests.test_gpu_track_f64_units import winding

NONE = np.zeros((0, 16))
FRAME = np.array([0.9, 0.02, 0.0, 0.6, 0.8, 0.0, 0.0, 0.0, 1.0])


def objective(ps, kl, p0, length, steps):
    ps = torch.from_numpy(ps)
    kq = (ps[:, 7] / ps[:, 6])[:, None]
    dt = (length / ps[:, 8] / steps)[:, None]

    def f(p, v):
        r = p[:, None, :] - p0[None]
        b = (torch.linalg.cross(kl[None].expand_as(r), r) / (r * r).sum(-1, keepdim=True) ** 1.5).sum(1)
        return v, kq * torch.linalg.cross(v, b)

    p, v = ps[:, 0:3], ps[:, 3:6]
    for _ in range(steps):
        a1, b1 = f(p, v)
        a2, b2 = f(p + dt / 2 * a1, v + dt / 2 * b1)
        a3, b3 = f(p + dt / 2 * a2, v + dt / 2 * b2)
        a4, b4 = f(p + dt * a3, v + dt * b3)
        p, v = p + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4), v + dt / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
    d = p - torch.from_numpy(FRAME[0:3])
    return ((d @ torch.from_numpy(FRAME[3:6])) ** 2 + (d @ torch.from_numpy(FRAME[6:9])) ** 2).mean()


@pytest.mark.parametrize("n_p,segments", [(1, [1]), (1, [31, 0, 129]), (3, [300]), (16, [127, 2049]), (17, [1000]),
                                          (33, [257]), (1, [20001]), (3, [9001]), (5, [8400]), (16, [9000]),
                                          (17, [9100]), (33, [9000, 0, 300])])
def test_gradient_matches_autograd(n_p, segments):
    ps = W.single_dipole_particles(n_p, seed=n_p)
    designs = [(*winding(s), NONE) for s in segments]
    # 3 steps: 12 stages of n_p points, a ragged last chunk of 256 for most n_p
    J, grad, _ = segment_gradient(engine.DesignSet(designs), ps, 0.0295, 0.01, np.tile(FRAME, (len(segments), 1)),
                                  checkpoint=2)
    at = 0
    for d, (kl, p0, _) in enumerate(designs):
        kl, p0 = torch.from_numpy(kl).requires_grad_(), torch.from_numpy(p0).requires_grad_()
        ref = objective(ps, kl, p0, 0.0295, 3)
        assert abs(J[d] - ref.item()) <= 1e-12 * ref.item()
        if len(kl):
            ref.backward()
            for got, want in ((grad[at:at + len(kl), 0:3], kl.grad.numpy()), (grad[at:at + len(kl), 3:6], p0.grad.numpy())):
                assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
        at += len(kl)


@pytest.mark.parametrize("part", [1.0, 0.5, 0.1, 0.06, 0.05, 0.04, 0.01])
def test_less_scratch(monkeypatch, part):
    """Less scratch than asked for: one pass, separate kernels, or the error, never another result."""
    from cctpy_gb300 import _lib

    lib = _lib.load()
    real = lib.cct_adjoint_scratch_bytes
    ds = engine.DesignSet([(*winding(20001), NONE)])
    ps = W.single_dipole_particles(16, seed=2)
    J, grad, _ = segment_gradient(ds, ps, 0.0295, 0.01, FRAME[None], checkpoint=2)
    monkeypatch.setattr(lib, "cct_adjoint_scratch_bytes", lambda *a: int(real(*a) * part))
    try:
        J2, grad2, _ = segment_gradient(ds, ps, 0.0295, 0.01, FRAME[None], checkpoint=2)
    except ValueError as e:
        assert "too small" in str(e) and part < 1.0
        return
    assert abs(J2[0] - J[0]) <= 1e-12 * J[0]
    assert np.linalg.norm(grad2 - grad) <= 1e-11 * np.linalg.norm(grad)
