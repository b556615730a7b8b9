"""A host allocation that fails inside an entry point is reported as a status and a message; it does not end the process."""
import subprocess
import sys

from tests.conftest import ROOT

CODE = """
import ctypes as C, resource
import numpy as np
from anechoic_b200 import _lib
L = _lib.load()
n, deg = 1000000, 20                       # a circulant graph: 80 MB of columns, the entry point's own copies need 500 MB
off = np.concatenate([np.arange(1, deg // 2 + 1), n - np.arange(1, deg // 2 + 1)[::-1]]).astype(np.int64)
col = np.ascontiguousarray(((np.arange(n, dtype=np.int64)[:, None] + off) % n).astype(np.int32))
rp = np.arange(0, n * deg + 1, deg, dtype=np.int32)
val = np.ones(n * deg, np.int8)
h = C.c_void_p()
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (200 << 20), resource.RLIM_INFINITY))
rc = L.anc_instance_create_csr(n, rp.ctypes.data, col.ctypes.data, val.ctypes.data, None, C.byref(h))
print(rc, L.anc_last_error().decode(), h.value)
"""


def test_failed_allocation_is_a_status(lib):
    p = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr[-500:])
    assert p.stdout.split("\n")[0] == "-2 out of host memory None"
