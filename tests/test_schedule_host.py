"""The schedule that cct_track takes (host only): owned, dataflow from 8 particle blocks on where a block
gets no CTA of its own or the estimate says so, grid barriers below that where the scratch is too small."""
import numpy as np
import pytest

from cctpy_gb300 import _lib
from cctpy_gb300.build import build_library

SMS, GRID, ROOM = 152, 456, 1 << 40


@pytest.fixture(scope="module")
def schedule():
    build_library()
    lib = _lib.load()

    def call(sizes, n_p, prec, scratch=ROOM):
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        return lib.cct_test_plan_schedule(off.ctypes.data, len(sizes), n_p, prec, SMS, GRID, scratch)

    return call


@pytest.mark.parametrize("prec", [0, 1])
def test_owned_dataflow_barriers(schedule, prec):
    assert schedule([46080], 2, prec) == 0
    assert schedule([46080] * 8, 2, prec) == 0
    assert schedule([600] * 160, 2, prec) == 1                 # more blocks than SMs
    assert schedule([597600], 4096, prec) == 1
    assert {schedule([46080], 16, prec, s) for s in range(256, 1 << 16, 256)} == {-1, 0, 2}
    assert schedule([46080], 16, prec, 256) == -1 and schedule([46080], 16, prec, 1 << 16) == 0


def test_bad_arguments(schedule):
    assert schedule([10], 0, 0) == -2 and schedule([10], 1, 2) == -2
    assert _lib.load().cct_test_plan_schedule(0, 1, 1, 0, SMS, GRID, ROOM) == -2
