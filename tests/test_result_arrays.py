"""The arrays that downloads come in are filled again only when
nothing refers to any of them (no GPU: the pool by itself)."""
from __future__ import annotations

import copy
import ctypes as C
import pickle
import threading
import weakref

import numpy as np
import pytest

NE, NN = 1 << 14, 17 ** 3 * 4   # arrays of 128 kB and above


def ids(dom):
    return [id(a) for a in dom.arrays()]


@pytest.fixture
def pool(pkg):
    p = pkg._ResultArrays()
    p.opened()
    return p


def test_a_dropped_result_is_filled_again(pool):
    d = pool.domain(NE, NN)
    first = ids(d)
    assert [a.size for a in d.arrays()] == [NN] * 6 + [NE] * 5
    assert all(a.flags.owndata and a.flags.writeable and a.dtype == np.float64 for a in d.arrays())
    del d
    assert ids(pool.domain(NE, NN)) == first


def test_a_chain_of_steps_takes_two_sets(pool):
    d, seen = pool.domain(NE, NN), set()
    for _ in range(10):
        new = pool.domain(NE, NN)
        assert not set(ids(new)) & set(ids(d))
        d = new
        seen.add(tuple(ids(d)))
        del new
    assert len(seen) == 2


# the array that is held, and by what
HOLDERS = {
    "record": ("e", lambda d: d),
    "copied record": ("p", lambda d: copy.copy(d)),
    "one array": ("q", lambda d: d.q),
    "last array": ("ss", lambda d: d.ss),
    "view": ("e", lambda d: d.e[2:5]),
    "reshaped": ("x", lambda d: d.x.reshape(17, -1)),
    "memoryview": ("v", lambda d: memoryview(d.v)),
    "ctypes": ("p", lambda d: d.p.ctypes),
    "pointer": ("p", lambda d: d.p.ctypes.data_as(C.c_void_p)),
    "buffer": ("xd", lambda d: C.c_double.from_buffer(d.xd)),
    "frombuffer": ("z", lambda d: np.frombuffer(d.z, dtype=np.float64)),
    "tensor": ("yd", lambda d: pytest.importorskip("torch").from_numpy(d.yd)),
    "closure": ("y", lambda d: (lambda a=d.y: a)),
    "cycle": ("zd", lambda d: (lambda l: l.append(l) or l)([d.zd])),
}


@pytest.mark.parametrize("how", HOLDERS)
def test_a_held_array_is_never_filled_again(pool, how):
    d = pool.domain(NE, NN)
    name, hold = HOLDERS[how]
    mine, held = id(getattr(d, name)), hold(d)   # alive from here on: no other array has its id
    del d
    for _ in range(3):
        one, two = pool.domain(NE, NN), pool.domain(NE, NN)
        assert mine not in ids(one) + ids(two)
        del one, two
    assert held is not None


def test_a_weak_reference_never_sees_another_step(pool):
    d = pool.domain(NE, NN)
    w = weakref.ref(d.e)
    del d
    for _ in range(3):
        d = pool.domain(NE, NN)
        assert w() is not d.e
        del d


def test_results_that_are_all_kept_by_the_caller(pool):
    kept = [pool.domain(NE, NN) for _ in range(20)]
    assert len({i for d in kept for i in ids(d)}) == 20 * 11
    for i, d in enumerate(kept):
        d.e[:] = i
    assert all(np.all(d.e == i) for i, d in enumerate(kept))
    assert len(pool._sets) <= pool.MOST_SETS


@pytest.mark.parametrize("ne", [1 << 14, 100 ** 3, 150 ** 3])
def test_what_is_kept_is_bounded(pool, ne):
    for k in range(8):
        pool.domain(ne + k, ne)
        assert len(pool._sets) <= pool.MOST_SETS
        assert sum(a.nbytes for s in pool._sets for a in s) <= pool.MOST_BYTES


def test_only_results_of_the_same_size(pool):
    a = pool.domain(NE, NN)
    first = ids(a)
    del a
    b = pool.domain(NE + 1, NN)
    assert b.e.size == NE + 1 and ids(b) != first
    assert ids(pool.domain(NE, NN)) == first


def test_small_arrays_are_not_kept(pool):
    pool.domain((1 << 14) - 1, 1 << 14)
    assert pool._sets == []


def test_all_is_given_back_with_the_last_context(pool):
    pool.opened()
    pool.domain(NE, NN)
    pool.closed()
    assert len(pool._sets) == 1
    pool.closed()
    assert pool._sets == []
    pool.domain(NE, NN)
    assert pool._sets == []


def test_threads_never_share_a_result(pool):
    """Each of several threads marks its result and finds the mark there."""
    wrong = []

    def work(me):
        for _ in range(300):
            d = pool.domain(NE, NN)
            d.e[0] = me
            d.ss[-1] = me
            if d.e[0] != me or d.ss[-1] != me:
                wrong.append(me)
            keep = d.p
            del d
            keep[0] = me
            if keep[0] != me:
                wrong.append(me)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_a_pickled_result_is_a_copy(pool):
    d = pool.domain(NE, NN)
    d.e[:] = 3.0
    back = pickle.loads(pickle.dumps(d.arrays()))
    del d
    pool.domain(NE, NN).e[:] = 4.0
    assert np.all(back[6] == 3.0)
