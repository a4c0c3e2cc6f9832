"""The arrays of a drop-in CSC call (api._csc_call), on a stand-in for the library:
a pattern of 3 columns and 4 entries behind a bound of 486 MB."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import ctypes as C, resource, sys
import numpy as np
from fortfem_b200 import _capi as K, api

calls = []

class Library:
    def __init__(self, status):
        self.status = status
    def entry(self, cap, nd, nz, cp, ri, val, st):
        calls.append(cap.value)
        nd._obj.value, nz._obj.value = 3, 4
        if self.status:
            st._obj.value = self.status
        elif cap.value < 4 or not cp:
            st._obj.value = K.FFG_CAPACITY
        else:
            C.memmove(cp, np.array([0, 1, 3, 4], np.int64).ctypes.data, 32)
            C.memmove(ri, np.array([0, 1, 2, 2], np.int32).ctypes.data, 16)
            C.memmove(val, np.array([1.0, 2.0, 3.0, 4.0]).ctypes.data, 32)
            st._obj.value = 0

def mapped():
    return int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()

limit, status = int(sys.argv[1]), int(sys.argv[2])
K.load = lambda: Library(status)
before = mapped()
if limit:
    resource.setrlimit(resource.RLIMIT_AS, (before + limit, before + limit))
A, st = api._csc_call("entry", [], "where", 20000, 45)
if status:
    assert A is None and st.code == status
else:
    assert st.code == 0 and A.nrow == 3
    assert list(A.col_ptr) == [0, 1, 3, 4] and list(A.row_idx) == [0, 1, 2, 2]
    assert list(A.val) == [1.0, 2.0, 3.0, 4.0]
    for a in (A.col_ptr, A.row_idx, A.val):
        assert a.base is None and a.flags.owndata
    assert mapped() - before < 100 << 20, mapped() - before
assert len(calls) == (2 if limit and not status else 1), calls
"""


@pytest.mark.parametrize("limit,status", [(0, 0), (64 << 20, 0), (0, -1), (64 << 20, -1)])
def test_csc_call_returns_what_it_does_not_need(limit, status):
    """The result's arrays hold the pattern alone; without the address space for the
    bound, the size is asked for; an error is the library's in both."""
    r = subprocess.run([sys.executable, "-c", CHILD, str(limit), str(status)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
