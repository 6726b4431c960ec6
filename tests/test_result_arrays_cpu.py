"""Result arrays in blocks of the library's pool own their memory, as every other new array does.  The pool here is a
stand-in with the C functions' signatures; the real one needs a GPU."""
import ctypes

import numpy as np
import pytest

from comet_b200 import _lib, api


class Pool:
    """Blocks of `room` bytes, `blocks` of them; counts what comes back."""

    def __init__(self, room, blocks):
        self.memory = [(ctypes.c_char * room)() for _ in range(blocks)]
        self.free = [ctypes.addressof(m) for m in self.memory]
        self.used, self.room = {}, room
        self.functions = {
            "comet_b200_result_alloc": ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_int64)(self.take),
            "comet_b200_result_size": ctypes.CFUNCTYPE(ctypes.c_int64, ctypes.c_void_p)(lambda p: self.used.get(p, 0)),
            "comet_b200_result_free": ctypes.CFUNCTYPE(None, ctypes.c_void_p)(self.give),
        }
        for name, fn in self.functions.items():
            setattr(self, name, fn)

    def take(self, n):
        if not self.free or n > self.room:
            return None
        p = self.free.pop()
        self.used[p] = self.room
        return p

    def give(self, p):
        assert self.used.pop(p, 0)
        self.free.append(p)


_ALL = []                      # arrays call their pool's functions when they go


@pytest.fixture
def pool(monkeypatch):
    p = Pool(1 << 20, 2)
    _ALL.append(p)
    monkeypatch.setattr(_lib, "load", lambda: p)
    monkeypatch.setattr(_lib, "address", lambda name: ctypes.cast(p.functions[name], ctypes.c_void_p).value)
    return p


@pytest.mark.parametrize("shape,dtype", [(40000, np.float64), ((300, 200), np.float64), (100000, np.int32), ((1, 1 << 17), np.float32)])
def test_results_own_their_memory(pool, shape, dtype):
    a, b = api._result(shape, dtype), api._result(shape, dtype)
    assert len(pool.used) == 2 and {a.ctypes.data, b.ctypes.data} == set(pool.used)
    for x in (a, b):
        assert x.flags.owndata and x.base is None and x.flags.c_contiguous and x.flags.writeable
        assert x.shape == (shape if isinstance(shape, tuple) else (shape,)) and x.dtype == dtype
    c = api._result(shape, dtype)                      # no block left: ordinary memory
    assert len(pool.used) == 2 and c.flags.owndata
    view = a[:10]
    del a
    assert len(pool.used) == 2                         # a view keeps its block
    del view, b, x
    assert not pool.used


def test_results_can_be_resized_in_place(pool):
    a = api._result(40000, np.float64)
    a[:] = np.arange(40000)
    p = a.ctypes.data
    a.resize(50000, refcheck=False)                    # still fits the block
    assert a.ctypes.data == p and np.array_equal(a[:40000], np.arange(40000)) and not a[40000:].any()
    a.resize(400000, refcheck=False)                   # does not: the block goes back
    assert not pool.used and np.array_equal(a[:40000], np.arange(40000)) and not a[40000:].any()
    a.resize(1000000, refcheck=False)
    assert np.array_equal(a[:40000], np.arange(40000))
    del a
    assert len(pool.free) == 2


def test_other_arrays_are_made_as_ever(pool):
    from numpy._core.multiarray import get_handler_name
    a = api._result(40000, np.float64)
    assert get_handler_name(a) == "comet_b200_results" and get_handler_name(np.empty(40000)) == "default_allocator"
    with pytest.raises(ValueError):
        api._result((40000, -1), np.float64)
    assert len(pool.used) == 1 and get_handler_name() == "default_allocator"
