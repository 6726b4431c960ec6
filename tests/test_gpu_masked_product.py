"""The masked product as dot products over the mask: list lengths at the edges of its kernels, every semiring, repeated
mask entries, rectangular operands, and operands that make it fall back to the push form."""
import numpy as np
import pytest

from comet_b200 import api
from oracle import oracle

pytestmark = pytest.mark.gpu


def _orc(t):
    return oracle.SparseArrays(t.format, t.nrows, t.ncols, t.a1pos, t.a1crd, t.a2pos, t.a2crd, t.val)


def _csr(rows, ncols, rng):
    pos = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    crd = np.concatenate([np.asarray(r, dtype=np.int64) for r in rows])
    return api.SparseTensor("CSR", len(rows), ncols, np.array([len(rows)]), np.array([-1]), pos, crd,
                            rng.uniform(0.5, 1.5, len(crd)))


def _pick(rng, n, k):
    return np.sort(rng.choice(n, k, replace=False))


def _check(A, B, M, semiring):
    got, ref = api.spgemm(A, B, M, semiring), oracle.spgemm(_orc(A), _orc(B), _orc(M), semiring)
    assert ref.val.shape[0] > 0
    assert np.array_equal(got.a2pos, ref.a2pos) and np.array_equal(got.a2crd, ref.a2crd)
    np.testing.assert_allclose(got.val, ref.val, rtol=1e-12)


@pytest.mark.parametrize("length", [1, 128, 129, 512, 513, 2048, 2049])
@pytest.mark.parametrize("longer", ["row of A", "column of B"])
@pytest.mark.parametrize("semiring", [api.PLUS_TIMES, api.PLUS_PAIR])
def test_list_lengths(length, longer, semiring):
    rng = np.random.default_rng(length)
    inner, short = 2500, max(1, min(length - 1, 90))
    a_len, b_len = (length, short) if longer == "row of A" else (short, length)
    A = _csr([_pick(rng, inner, a_len) if i % 6 else _pick(rng, inner, 7) for i in range(70)], inner, rng)
    cols = [_pick(rng, inner, b_len if j % 5 else 40) for j in range(150)]            # columns of B
    rows = [[] for _ in range(inner)]
    for j, c in enumerate(cols):
        for k in c:
            rows[k].append(j)
    B = _csr(rows, 150, rng)
    M = _csr([_pick(rng, 150, 1 + i) for i in range(70)], 150, rng)
    _check(A, B, M, semiring)


@pytest.mark.parametrize("semiring", range(8))
def test_every_semiring_and_repeated_mask_entries(semiring):
    rng = np.random.default_rng(semiring)
    n = 700
    A = _csr([_pick(rng, n, int(k)) for k in rng.integers(0, 300, n)], n, rng)
    B = _csr([_pick(rng, n, int(k)) for k in rng.integers(0, 200, n)], n, rng)
    M = _csr([np.sort(rng.integers(0, n, int(k))) for k in rng.integers(0, 90, n)], n, rng)
    _check(A, B, M, semiring)


@pytest.mark.parametrize("which", ["unordered B", "repeats in A", "repeats in B", "dense mask"])
def test_operands_for_the_push_form(which):
    rng = np.random.default_rng(3)
    n = 400
    rows = lambda make: _csr([make() for _ in range(n)], n, rng)
    A = rows(lambda: np.sort(rng.integers(0, n, 40)) if which == "repeats in A" else _pick(rng, n, 3 if which == "dense mask" else 40))
    B = rows(lambda: rng.permutation(n)[:30] if which == "unordered B"
             else np.sort(rng.integers(0, n, 30)) if which == "repeats in B" else _pick(rng, n, 2 if which == "dense mask" else 30))
    M = rows(lambda: _pick(rng, n, 390 if which == "dense mask" else 50))
    for semiring in (api.PLUS_TIMES, api.PLUS_PAIR, api.MIN_PLUS):
        _check(A, B, M, semiring)
