"""Field calls whose workspace cannot be had, or does not match the design."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from cctpy_gb300 import _lib, engine
from tests.test_gpu_field_split import points, winding

NONE = np.zeros((0, 16))


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
