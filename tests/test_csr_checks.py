"""CSR couplings are checked before anything reaches the device: rows in any order are taken, asymmetric values, missing or
surplus mirror entries and duplicates are refused with the same messages whatever the order of the rows."""
import ctypes as C

import numpy as np
import pytest

from anechoic_b200 import _lib


def _create(rows):
    """rows: list of [(col, val), ...]; returns (status, message)."""
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    col = np.array([c for r in rows for c, _ in r], np.int32)
    val = np.array([v for r in rows for _, v in r], np.int8)
    L, h = _lib.load(), C.c_void_p()
    rc = L.anc_instance_create_csr(len(rows), rp.ctypes.data, col.ctypes.data, val.ctypes.data, None, C.byref(h))
    msg = L.anc_last_error().decode()
    if h.value:
        L.anc_instance_destroy(h)
    return rc, msg


GOOD = [[(3, 2), (1, -1)], [(0, -1), (2, 1)], [(1, 1)], [(0, 2)]]


def test_rows_in_any_order_pass_the_checks():
    for rows in (GOOD, [sorted(r) for r in GOOD], [[], []]):
        rc, msg = _create(rows)
        assert rc in (_lib.ANC_OK, _lib.ANC_ECUDA), msg          # without a GPU the upload is what fails


@pytest.mark.parametrize("rows,message", [
    ([[(1, 1)], [(0, -1)]], "not symmetric"),
    ([[(1, 1)], []], "not symmetric"),
    ([[(2, 1), (1, 1)], [(0, 1)], [(0, 1), (1, 1)]], "not symmetric"),
    ([[(1, 1), (1, 1)], [(0, 1)]], "not symmetric"),
    ([[(1, 1), (1, 1)], [(0, 1), (0, 1)]], "duplicate"),
    ([[(1, 1), (2, 1), (1, 2)], [(0, 2), (0, 1)], [(0, 1)]], "duplicate"),
])
def test_refused(rows, message):
    rc, msg = _create(rows)
    assert rc == _lib.ANC_EINVAL and message in msg
