"""cct_track_copied with more particles than the host's memory holds: an error, not the end of the process."""
import os
import subprocess
import sys

from cctpy_gb300 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CALL = """
import ctypes
from cctpy_gb300 import _lib
lib = _lib.load()
off = (ctypes.c_int64 * 2)(0, 1)
one = (ctypes.c_double * 10)()
at = ctypes.addressof
n = 110_000_000_000_000_000          # 8.8e18 bytes
rc = lib.cct_track_copied(0, 0, at(off), at(off), 0, 0, at(off), 1, at(one), 1, at(one), n, 1.0, 1.0, 0, 256, 2 ** 63 - 1,
                          256, 256, 0)
print(rc, _lib.last_error())
"""


def test_no_host_memory():
    r = subprocess.run([sys.executable, "-c", CALL], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert r.stdout.startswith(f"{_lib.CCT_ERR_CUDA} ") and "host memory" in r.stdout
