"""Host arrays are looked at page by page before a kernel reads them: a hole in the
middle of one has to end the process on the host (here a child), whole arrays not."""
import os
import signal
import subprocess
import sys

import pytest

import cumetis_gb300 as cm
from conftest import ROOT

CHILD = r"""
import ctypes, mmap, resource, sys
lib = ctypes.CDLL(sys.argv[1])
touch = lib._Z14cm_touch_pagesPKvm
touch.argtypes, touch.restype = [ctypes.c_void_p, ctypes.c_size_t], None
first, bytes_, hole = (int(x) for x in sys.argv[2:5])
resource.setrlimit(resource.RLIMIT_CORE, (0, 0))
page = mmap.PAGESIZE
m = mmap.mmap(-1, 16 * page)
base = ctypes.addressof(ctypes.c_char.from_buffer(m))
if hole >= 0:
    libc = ctypes.CDLL(None, use_errno=True)
    libc.mprotect.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]
    assert libc.mprotect(base + hole * page, page, 0) == 0
units = lambda x: (x // 10) * page + x % 10  # pages * 10 + bytes
touch(base + units(first), units(bytes_))
print("whole")
"""


@pytest.mark.parametrize("first,size,hole,ends", [
    (0, 160, -1, False), (0, 0, 0, False), (4, 1, 1, False), (0, 70, 7, False), (80, 80, 7, False), (4, 14, 2, False),
    (0, 160, 0, True), (0, 160, 7, True), (0, 160, 15, True), (4, 24, 2, True), (68, 12, 7, True), (0, 71, 7, True)])
def test_touch(tmp_path, first, size, hole, ends):
    cm.lib()
    lib = os.path.join(ROOT, "cumetis_gb300", "libcm.so")
    r = subprocess.run([sys.executable, "-c", CHILD, lib, str(first), str(size), str(hole)], stdout=subprocess.PIPE,
                       stderr=subprocess.PIPE, cwd=tmp_path)
    if ends:
        assert r.returncode == -signal.SIGSEGV and b"whole" not in r.stdout
    else:
        assert r.returncode == 0 and b"whole" in r.stdout, r.stderr
