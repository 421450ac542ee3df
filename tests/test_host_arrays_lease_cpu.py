"""The memory of build results goes back by itself when its last user is gone, whatever an interpreter's
reference counts look like (one that passes locals as borrowed references counts one less)."""
import gc
import sys
import threading
import weakref

import numpy as np
import pytest

from bvh_gb300 import NODE_DTYPE
from bvh_gb300.builders import _HostArrays


def _at(a):
    return a.ctypes.data


@pytest.fixture(params=[0, -1])
def counts(request, monkeypatch):
    real = sys.getrefcount
    monkeypatch.setattr(sys, "getrefcount", lambda x: real(x) - 1 + request.param)  # (one frame more: this one)


def test_held_memory_is_not_handed_out(counts):
    h = _HostArrays()
    held = h.take(NODE_DTYPE, 50_000)
    held["left"] = 5
    for _ in range(4):
        other = h.take(NODE_DTYPE, 50_000)
        assert not np.shares_memory(held, other)
        other["left"] = 6
    assert (held["left"] == 5).all()


@pytest.mark.parametrize("keeper", [lambda a: a[10:20], lambda a: a.view(np.uint8), lambda a: memoryview(a),
                                    lambda a: a["left"].T, lambda a: [a], lambda a: np.frombuffer(a, np.uint8)])
def test_every_kind_of_view_holds_the_memory(counts, keeper):
    h = _HostArrays()
    a = h.take(NODE_DTYPE, 50_000)
    at, kept = _at(a), keeper(a)
    del a
    gc.collect()
    other = h.take(NODE_DTYPE, 50_000)
    assert _at(other) != at
    del kept
    gc.collect()
    again = h.take(NODE_DTYPE, 50_000)
    assert _at(again) == at and again.flags.writeable and again.dtype == NODE_DTYPE


def test_threads_never_share():
    h = _HostArrays()
    wrong = []

    def work(k):
        for i in range(200):
            a = h.take(np.uint32, 300_000)
            a[::5000] = k * 1000 + i
            b = a[::5000]
            del a
            if not (b == k * 1000 + i).all():
                wrong.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not wrong


def test_idle_limit_and_closed_pool():
    h = _HostArrays(keep=2)
    held = [h.take(np.uint32, 300_000 + k) for k in range(20)]
    memory = [weakref.ref(m) for m, _ in h._pieces]
    assert all(m() is not None for m in memory)
    while held:  # as results are dropped, their memory goes, not only at the next build
        held.pop()
    gc.collect()
    assert sum(m() is not None for m in memory) <= 2 + 4  # the idle ones that stay, and two results as always
    last = h.take(np.uint32, 300_000)
    del h
    last[:] = 1  # outlives its pool
    assert last.sum() == 300_000
