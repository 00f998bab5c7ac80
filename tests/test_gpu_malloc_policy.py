"""Creating a context or a batch leaves the process's allocator alone: a block
that the C library maps on its own before is mapped on its own after.  In a
process of its own, whose allocator nothing else has adapted."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import __graft_entry__ as ge
libc = C.CDLL(None)
if not hasattr(libc, "mallinfo2"):
    sys.exit(77)
class Info(C.Structure):
    _fields_ = [(k, C.c_size_t) for k in ("arena ordblks smblks hblks hblkhd usmblks fsmblks uordblks fordblks keepcost").split()]
libc.mallinfo2.restype = Info
libc.malloc.restype, libc.malloc.argtypes = C.c_void_p, [C.c_size_t]
libc.free.argtypes = [C.c_void_p]
def mapped():
    before = libc.mallinfo2().hblks
    p = libc.malloc(24 << 20)
    after = libc.mallinfo2().hblks
    # not given back: freeing a mapped block is what raises the threshold
    return after - before
pkg = ge.load_package()
with pkg.Lulesh(3) as g:
    g.run(1)
first = mapped()
with pkg.Lulesh(30), pkg.Batch([30, 28]):
    pass
print(first, mapped())
"""


def test_large_blocks_are_mapped_as_before(pkg):
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    if r.returncode == 77:
        pytest.skip("no mallinfo2")
    assert r.returncode == 0, r.stderr
    first, second = r.stdout.split()[-2:]
    assert first == second, r.stdout
