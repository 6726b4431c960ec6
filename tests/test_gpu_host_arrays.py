"""Host arrays in and out: sizes at the edges of the staged copies (driver copy, one piece, several pieces, several
chunks), sources at odd addresses, and result arrays from the page-locked pool."""
import time

import numpy as np
import pytest
import torch

from comet_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 12287, 12288, 12289, 65536, 65537, 262143, 270000, 2200000])
@pytest.mark.parametrize("offset", [0, 3])
def test_coordinates_of_every_size_come_back_sorted(n, offset):
    rng = np.random.default_rng(n + offset)
    rows, cols = rng.integers(0, 5000, n + offset)[offset:], rng.integers(0, 7001, n + offset)[offset:]
    vals = rng.uniform(-1, 1, n + offset)[offset:]
    C = api.from_coordinates(rows, cols, vals, (5000, 7001))
    order = np.lexsort((np.arange(n), cols, rows))
    assert np.array_equal(C.a2pos, np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=5000))]))
    assert np.array_equal(C.a2crd, cols[order]) and np.array_equal(C.val, vals[order])


def test_results_that_are_kept_do_not_share_memory():
    """More results alive than the pool has blocks for, each of them right, then blocks taken again."""
    A = api.SparseTensor("CSR", 40000, 40000, np.array([40000]), np.array([-1]), np.arange(40001), np.arange(40000),
                         np.ones(40000))
    kept = []
    for i in range(12):
        x = np.full(40000, float(i))
        kept.append(api.spmv(A, x))
        if i % 5 == 4:
            torch.cuda.synchronize()
    for i, y in enumerate(kept):
        assert np.array_equal(y, np.full(40000, float(i)))
    view = kept[3][100:200]
    del kept, y
    assert np.array_equal(view, np.full(100, 3.0))          # a view keeps its block
    for i in range(4):
        assert np.array_equal(api.spmv(A, np.full(40000, 7.0 + i)), np.full(40000, 7.0 + i))
    assert np.array_equal(view, np.full(100, 3.0))
    _lib.load().comet_b200_release_scratch()
    assert np.array_equal(view, np.full(100, 3.0))
    assert np.array_equal(api.spmv(A, np.full(40000, 2.0)), np.full(40000, 2.0))


@pytest.mark.parametrize("shape", [(1, 1), (1, 70000), (70000, 1), (3, 1 << 40), (1 << 20, 1 << 12)])
@pytest.mark.parametrize("n", [4095, 4096, 4097, 40000])
def test_sort_keys_of_every_width(shape, n):
    """One digit, keys of up to 32 bits, wider ones; tiles of 4096 keys."""
    rng = np.random.default_rng(n)
    rows, cols = rng.integers(0, shape[0], n), rng.integers(0, shape[1], n)
    cols[::3] = cols[0]
    vals = rng.uniform(-1, 1, n)
    C = api.from_coordinates(rows, cols, vals, shape)
    order = np.lexsort((np.arange(n), cols, rows))
    assert np.array_equal(C.a2pos, np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=shape[0]))]))
    assert np.array_equal(C.a2crd, cols[order]) and np.array_equal(C.val, vals[order])


def test_results_from_the_pool_own_their_memory_and_can_be_resized():
    A = api.SparseTensor("CSR", 60000, 60000, np.array([60000]), np.array([-1]), np.arange(60001), np.arange(60000),
                         np.ones(60000))
    x = np.arange(60000.0)
    lib, ys = _lib.load(), []
    for _ in range(400):                                    # the pool makes its blocks in the background
        ys.append(api.spmv(A, x))
        if lib.comet_b200_result_size(ys[-1].ctypes.data):
            break
        ys = ys[-1:]
        time.sleep(0.005)
    else:
        pytest.fail("no result came from the pool")
    y = ys.pop()
    assert y.flags.owndata and y.base is None and np.array_equal(y, x)
    p = y.ctypes.data
    y.resize(200000, refcheck=False)
    assert np.array_equal(y[:60000], x) and not y[60000:].any() and lib.comet_b200_result_size(p) == 0
