"""The memory that build results lie in: reused once nobody refers to it, never before."""
import gc

import numpy as np

from bvh_gb300 import NODE_DTYPE
from bvh_gb300.builders import _HostArrays


def _at(a):
    return a.ctypes.data


def test_reused_only_when_unreferenced():
    h = _HostArrays()
    a = h.take(NODE_DTYPE, 100_000)
    a["left"] = 7
    b = h.take(NODE_DTYPE, 100_000)
    assert _at(a) != _at(b)
    first = _at(a)
    view = a["min"][5:50]  # any view keeps the memory
    del a
    c = h.take(NODE_DTYPE, 100_000)
    assert _at(c) not in (first, _at(b))
    assert (view.base is not None) and _at(view) == first + 5 * 48
    del view
    gc.collect()
    d = h.take(NODE_DTYPE, 100_000)
    assert _at(d) == first
    assert len({_at(x) for x in (b, c, d)}) == 3


def test_arrays_of_other_objects_keep_it():
    h = _HostArrays()
    a = h.take(np.uint32, 400_000)
    m = memoryview(a)
    at = _at(a)
    del a
    b = h.take(np.uint32, 400_000)
    assert _at(b) != at
    m.release()
    del m, b
    assert _at(h.take(np.uint32, 400_000)) is not None


def test_bounded_and_sized():
    h = _HostArrays(keep=2)
    held = [h.take(np.uint32, 300_000 + k) for k in range(6)]
    del held
    small = h.take(np.uint32, 300_000)
    assert len(h._pieces) <= 4  # two idle ones, the one in use, the last one made
    big = h.take(np.uint32, 3_000_000)
    assert big.size == 3_000_000 and small.size == 300_000
    at = _at(big)
    del big
    tiny = h.take(np.uint32, 300_000)  # ten times too large a piece is not taken
    assert _at(tiny) != at
    assert h.take(np.uint32, 10).size == 10 and h.take(np.uint32, 0).size == 0
