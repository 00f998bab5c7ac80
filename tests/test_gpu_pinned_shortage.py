"""No pinned memory for the buffer that small states pass through: contexts
are created and work all the same, their arrays copied one by one.  The
shortage is a preloaded function that fails allocations of the buffer's size."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static void *real_one(const char *name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }
static int fails(size_t n) { return n > 40000; }   /* the state of s = 8: 55,472 bytes */
int cudaHostAlloc(void **p, size_t n, unsigned flags)
{
    int (*real)(void **, size_t, unsigned) = (int (*)(void **, size_t, unsigned))real_one("cudaHostAlloc");
    return fails(n) ? 2 : real(p, n, flags);
}
int cudaMallocHost(void **p, size_t n)
{
    int (*real)(void **, size_t) = (int (*)(void **, size_t))real_one("cudaMallocHost");
    return fails(n) ? 2 : real(p, n);
}
"""

CHILD = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
import __graft_entry__ as ge
pkg = ge.load_package()
with pkg.Lulesh(8) as g, pkg.Lulesh(8) as ref:
    d = g.download()
    for _ in range(4):
        d = pkg.lulesh(g, d)
    ref.run(4)
    for k in ("x", "xd", "e", "v"):
        assert np.array_equal(g.get_field(k), getattr(d, k)), k
        assert np.array_equal(ref.get_field(k), getattr(d, k)), k
print("worked")
"""


def test_contexts_without_the_pinned_buffer(pkg, tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=str(ROOT))], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": str(so)})
    assert r.returncode == 0 and "worked" in r.stdout, r.stdout + r.stderr
