"""The masked count holds the longer of M_i and B_k as a set and streams the other.  Set lengths at the edges of its
three kernels, both sides, column spaces wider than one bitmap, and operands that rule a side out."""
import numpy as np
import pytest

from comet_b200 import api
from oracle import oracle

pytestmark = pytest.mark.gpu


def _orc(t):
    return oracle.SparseArrays(t.format, t.nrows, t.ncols, t.a1pos, t.a1crd, t.a2pos, t.a2crd, t.val)


def _csr(rows, ncols):
    """CSR of a list of coordinate arrays, in the order given."""
    pos = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    crd = np.concatenate([np.asarray(r, dtype=np.int64) for r in rows]) if pos[-1] else np.zeros(0, np.int64)
    return api.SparseTensor("CSR", len(rows), ncols, np.array([len(rows)]), np.array([-1]), pos, crd, np.ones(len(crd)))


def _pick(rng, n, k):
    return np.sort(rng.choice(n, k, replace=False))


def _check(A, B, M):
    want = oracle.masked_pair_count(_orc(A), _orc(B), _orc(M))
    assert want > 0
    assert api.masked_pair_count(A, B, M) == want


@pytest.mark.parametrize("length", [1, 127, 128, 129, 512, 513, 2048, 2049, 6000])
@pytest.mark.parametrize("side", ["mask", "b"])
def test_set_lengths(length, side):
    rng = np.random.default_rng(length)
    n, short = 7000, max(1, min(length - 1, 100))
    m_len, b_len = (length, short) if side == "mask" else (short, length)
    M = _csr([_pick(rng, n, m_len) if i % 7 else [] for i in range(60)], n)
    B = _csr([_pick(rng, n, b_len) if k % 5 else _pick(rng, n, 33) for k in range(n)], n)
    A = _csr([_pick(rng, n, 1 + 11 * i) for i in range(60)], n)
    _check(A, B, M)


@pytest.mark.parametrize("stored", [1400000, 1500001, 3100000])      # columns that M stores, of 4 million
def test_column_space_wider_than_one_bitmap(stored):
    rng = np.random.default_rng(5)
    n = 4000000
    used = _pick(rng, n, stored)
    M = _csr([used] + [rng.permutation(used)[:k] for k in (3, 200, 700)] + [_pick(rng, n, 9)], n)
    for i in range(5):
        M.a2crd[M.a2pos[i]:M.a2pos[i + 1]].sort()
    B = _csr([_pick(rng, n, k) for k in (5, 150, 600, 3000, 40000)] + [used[::3]], n)
    A = _csr([np.arange(6)] * 5, 6)
    _check(A, B, M)


def test_operands_that_rule_a_side_out():
    rng = np.random.default_rng(9)
    n = 3000
    A = _csr([_pick(rng, n, 40) for _ in range(200)], n)
    M = _csr([_pick(rng, n, 60) for _ in range(200)], n)
    unordered = _csr([rng.permutation(_pick(rng, n, 300 + 400 * (k % 2))) for k in range(n)], n)
    _check(A, unordered, M)
    repeats = _csr([np.sort(rng.integers(0, n, 300 + 400 * (k % 2))) for k in range(n)], n)
    _check(A, repeats, M)
    _check(A, repeats, _csr([np.sort(rng.integers(0, n, 60)) for _ in range(200)], n))     # M repeats coordinates
    tall = _csr([_pick(rng, 500, 200) for _ in range(n)], 500)                              # more rows of B than columns
    _check(A, tall, _csr([_pick(rng, 500, 60) for _ in range(200)], 500))
