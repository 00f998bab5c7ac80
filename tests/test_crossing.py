"""The choice of how a Domain record's arrays cross between host and device
(csrc/crossing.h), compiled for the host and asked about arrays that a kernel
must not be given.  No GPU: the wrong choice would fault one."""
from __future__ import annotations

import ctypes as C
import subprocess

import pytest

from conftest import ROOT

PAGEABLE, PINNED, OTHER = range(3)
STAGED, DIRECT, COPIED = range(3)

SOURCE = """
#include "crossing.h"
extern "C" int choose(const lulesh::HostArray *a, int n, int to_host, int buffer)
{
    return static_cast<int>(lulesh::crossing(a, n, to_host != 0, buffer != 0));
}
"""


class HostArray(C.Structure):
    _fields_ = [("at", C.c_size_t), ("bytes", C.c_size_t), ("memory", C.c_int), ("device", C.c_size_t),
                ("piece", C.c_size_t), ("piece_bytes", C.c_size_t), ("writable", C.c_bool)]


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("crossing")
    (d / "c.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "lulesh-accelerate_gb300" / "csrc"),
                    str(d / "c.cpp"), "-o", str(d / "c.so")], check=True)
    lib = C.CDLL(str(d / "c.so"))

    def call(arrays, to_host=False, buffer=True):
        return lib.choose((HostArray * len(arrays))(*arrays), len(arrays), int(to_host), int(buffer))
    return call


def pinned(at=0x10000, n=100, **over):
    """An array of n values in a pinned piece of its own."""
    a = HostArray(at, 8 * n, PINNED, at, at, 8 * n, True)
    for k, v in over.items():
        setattr(a, k, v)
    return a


def record(change=None, at=4):
    """Eleven pinned arrays, one of them changed."""
    a = [pinned(0x10000 * (i + 1)) for i in range(11)]
    if change is not None:
        a[at] = change(a[at])
    return a


def change(**over):
    def f(a):
        for k, v in over.items():
            setattr(a, k, v(a) if callable(v) else v)
        return a
    return f


@pytest.mark.parametrize("to_host", [False, True])
@pytest.mark.parametrize("buffer", [False, True])
def test_whole_pinned_arrays_are_read_and_written_by_the_kernel(choose, to_host, buffer):
    assert choose(record(), to_host, buffer) == DIRECT
    assert choose(record(change(at=0)), to_host, buffer) == DIRECT          # one left out
    inside = change(piece=lambda a: a.at - 64, piece_bytes=lambda a: a.bytes + 128)
    assert choose(record(inside), to_host, buffer) == DIRECT
    tail = change(piece=lambda a: a.at - 64, piece_bytes=lambda a: a.bytes + 64)
    assert choose(record(tail), to_host, buffer) == DIRECT


@pytest.mark.parametrize("at", [0, 5, 6, 10])
@pytest.mark.parametrize("to_host", [False, True])
@pytest.mark.parametrize("over", [
    dict(at=lambda a: a.at + 4, device=lambda a: a.device + 4, bytes=lambda a: a.bytes - 8),   # not on a word
    dict(at=lambda a: a.at + 1, device=lambda a: a.device + 1, bytes=lambda a: a.bytes - 8),
    dict(device=lambda a: a.device + 4),
    dict(device=0),                                             # not mapped
    dict(piece=0, piece_bytes=0),                               # extent not known
    dict(piece_bytes=lambda a: a.bytes - 8),                    # ends one value early
    dict(piece_bytes=8),                                        # a piece at each end, a gap between
    dict(piece=lambda a: a.at + 8),                             # begins one value late
    dict(piece=lambda a: a.at - 64, piece_bytes=lambda a: a.bytes + 56),
    dict(piece=lambda a: a.at - 4096, piece_bytes=4096),        # the piece before
])
def test_arrays_a_kernel_cannot_take_are_copied(choose, over, to_host, at):
    assert choose(record(change(**over), at), to_host) == COPIED


def test_arrays_a_kernel_cannot_write(choose):
    assert choose(record(change(writable=False)), to_host=True) == COPIED
    assert choose(record(change(writable=False)), to_host=False) == DIRECT


@pytest.mark.parametrize("shift", [0, 8, 792, -8])
def test_arrays_that_share_memory(choose, shift):
    """Copies to them come one after the other; a kernel's stores do not."""
    a = record()
    a[9] = pinned(a[2].at, piece=a[2].at - 4096, piece_bytes=8192)
    a[9].at += shift
    a[9].device += shift
    assert choose(a, to_host=True) == COPIED
    assert choose(a, to_host=False) == DIRECT
    a[9].at = 0
    assert choose(a, to_host=True) == DIRECT


@pytest.mark.parametrize("to_host", [False, True])
def test_memory_that_is_not_the_hosts_never_meets_memcpy(choose, to_host):
    """A device or managed array among pageable or pinned ones, in either
    order: the copies tell what they cannot take."""
    for other in (0, 4, 10):
        for page in (None, 0, 4, 10):
            a = record(change(memory=OTHER), other)
            if page is not None and page != other:
                a[page].memory = PAGEABLE
            assert choose(a, to_host) == COPIED


@pytest.mark.parametrize("to_host", [False, True])
def test_pageable_arrays(choose, to_host):
    """Any pageable one: through the buffer where there is one, whatever the
    alignment or extent of the pinned ones among them."""
    for a in (record(change(memory=PAGEABLE)), [pinned(memory=PAGEABLE, at=0x10001 + 0x10000 * i) for i in range(11)]):
        assert choose(a, to_host, True) == STAGED
        assert choose(a, to_host, False) == COPIED
    a = record(change(memory=PAGEABLE))
    a[7].piece_bytes = 8
    assert choose(a, to_host, True) == STAGED
    assert choose(a, to_host, False) == COPIED
