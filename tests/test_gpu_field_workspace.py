"""Field calls whose workspace cannot be had, or does not match the design."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import _lib, engine
from tests.test_gpu_field_split import points, winding

NONE = np.zeros((0, 16))


@pytest.mark.parametrize("prec", ["f64", "f32c"])
@pytest.mark.parametrize("n", [5, 700])
def test_no_memory_for_a_workspace(monkeypatch, prec, n):
    """A nearly full GPU (the workspace's allocation fails): the same fields, unsplit."""
    ds = engine.DesignSet([(*winding(6000), NONE)])
    pts = points(n, 3)
    want = engine.field_at_points(ds, pts, prec)
    ds.packed()
    empty = torch.empty

    def full(*a, **k):
        if k.get("dtype") is torch.uint8 and int(a[0]) > 48 * n:
            raise torch.OutOfMemoryError("out of memory")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    assert np.array_equal(engine.field_at_points(ds, pts, prec), want)
    assert np.array_equal(engine.field_at_points(ds, torch.from_numpy(pts).cuda(), prec).cpu().numpy(), want)


def test_fewer_segments_than_the_design_has():
    ds = engine.DesignSet([(*winding(6000), NONE)])
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    engine.field_status()
    for n in (3, 500):
        pts = torch.from_numpy(points(n, 3)).cuda()
        out = torch.empty_like(pts)
        nbytes = lib.cct_field_work_bytes(1000, n, 1)
        assert nbytes > 0
        work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        _lib.check(lib.cct_field_f32c_ws(ds.packed().data_ptr(), 0, 1000, 0, 0, pts.data_ptr(), n, out.data_ptr(),
                                         work.data_ptr(), nbytes, st), "field")
        assert torch.isnan(out).all()
        with pytest.raises(ValueError):
            engine.field_status()
        engine.field_status()
