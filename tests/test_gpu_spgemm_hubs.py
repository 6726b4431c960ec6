"""Products whose long rows of B are ORed into the bitmaps as a whole: rows of B at the limits, more of them in a row of A than a
list holds, repeated columns, columns that B does not store, both folds, bitmaps kept and not kept."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402

pytestmark = pytest.mark.gpu


def _csr(rows, vals, shape):
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    m = sp.csr_matrix(shape)
    m.indptr, m.indices, m.data = ptr, np.concatenate(rows), vals
    return m


def _device(m):
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return dev.DeviceCSR(*m.shape, up(m.indptr.astype(np.int64)), up(m.indices.astype(np.int64)), up(m.data))


def _operands(ncols, step, repeats):
    """2600 rows of B in the columns that `step` divides: 1400 long ones, lengths around 512 and around an eighth of the words."""
    rng = np.random.default_rng(3)
    stored = np.arange(0, ncols, step)
    edge = max(512, (stored.size + 31) // 32 // 8)
    lens = [511, 512, 513, edge - 1, edge, edge + 1, 1024, 1025, stored.size] + list(rng.integers(520, 700, 1391)) + list(rng.integers(0, 60, 1200))
    brows = [np.sort(rng.choice(stored, min(n, stored.size), replace=False)) for n in lens]
    if repeats:
        brows[7][1::2] = brows[7][::2][:brows[7][1::2].size]
    B = _csr(brows, rng.uniform(0.5, 1, sum(map(len, brows))), (len(brows), ncols))
    n = len(brows)
    arows = [np.array([0, 1]), np.array([1, 2]), np.arange(9), np.array([8]), np.arange(n), np.arange(0, n, 2), np.arange(1400, n),
             np.concatenate([np.arange(513), np.arange(1400, n)]), np.arange(1025), np.array([], dtype=int)]
    arows += [np.sort(rng.choice(n, 30, replace=False)) for _ in range(2990)]
    A = _csr(arows, rng.uniform(-1, 1, sum(map(len, arows))), (len(arows), n))
    return A, B


@pytest.mark.parametrize("semiring", [api.PLUS_TIMES, api.MIN_PLUS])
@pytest.mark.parametrize("ncols,step", [(200001, 1), (262144, 3), (819200, 1), (819232, 1), (900000, 2), (300000, 60000)])
def test_long_rows_of_b(ncols, step, semiring, monkeypatch):
    if semiring == api.MIN_PLUS:
        monkeypatch.setenv("COMET_B200_SPGEMM_BITMAP_GB", "0")
    A, B = _operands(ncols, step, repeats=step == 3)
    C = dev.spgemm(_device(A), _device(B), semiring=semiring)
    pos, crd, val = C.pos.cpu().numpy(), C.crd.cpu().numpy(), C.val.cpu().numpy()
    want = sp.csr_matrix((np.ones(A.nnz), A.indices, A.indptr), A.shape) @ sp.csr_matrix((np.ones(B.nnz), B.indices, B.indptr), B.shape)
    want.sort_indices()
    assert np.array_equal(pos, want.indptr) and np.array_equal(crd, want.indices)
    if semiring == api.PLUS_TIMES:
        ref, mag = A @ B, abs(A) @ abs(B)
        ref.sort_indices(), mag.sort_indices()
        # a sum of n products in any order: n * 2^-53 of the sum of their magnitudes, n up to 2600
        assert np.all(np.abs(val - ref.data) <= 2600 * 2.0 ** -53 * mag.data)
    else:
        for r in list(range(10)) + list(range(10, A.shape[0], 97)):
            out = np.full(ncols, np.inf)
            for k, a in zip(A.indices[A.indptr[r]:A.indptr[r + 1]], A.data[A.indptr[r]:A.indptr[r + 1]]):
                b = slice(B.indptr[k], B.indptr[k + 1])
                np.minimum.at(out, B.indices[b], a + B.data[b])
            assert np.array_equal(val[pos[r]:pos[r + 1]], out[crd[pos[r]:pos[r + 1]]])


@pytest.mark.parametrize("stored", [146000, 240000, 262000])
def test_rows_with_more_columns_than_the_stage_holds(stored):
    """Columns that need a look-up, rows of 32 words with from a few to all of their 1024 columns: staged, word by word, and both in turn."""
    rng = np.random.default_rng(stored)
    columns = np.sort(rng.choice(300000, stored, replace=False))
    brows = [np.sort(rng.choice(columns, 600, replace=False)) for _ in range(400)]
    brows[0] = columns                                                    # all of them are stored
    brows += [columns[:7000], columns[3000:3400], columns[-2000:]]
    B = _csr(brows, rng.uniform(0.5, 1, sum(map(len, brows))), (len(brows), 300000))
    arows = [np.sort(rng.choice(np.arange(1, 403), n, replace=False)) for n in (40, 80, 110, 130, 160, 200, 300, 402) * 6]
    arows += [np.array([0]), np.array([400, 401, 402])] + [np.sort(rng.choice(np.arange(1, 400), 2, replace=False)) for _ in range(1900)]
    A = _csr(arows, rng.uniform(-1, 1, sum(map(len, arows))), (len(arows), len(brows)))
    C = dev.spgemm(_device(A), _device(B))
    pos, crd, val = C.pos.cpu().numpy(), C.crd.cpu().numpy(), C.val.cpu().numpy()
    want = sp.csr_matrix((np.ones(A.nnz), A.indices, A.indptr), A.shape) @ sp.csr_matrix((np.ones(B.nnz), B.indices, B.indptr), B.shape)
    ref, mag = A @ B, abs(A) @ abs(B)
    want.sort_indices(), ref.sort_indices(), mag.sort_indices()
    assert np.array_equal(pos, want.indptr) and np.array_equal(crd, want.indices)
    # a sum of n products in any order: n * 2^-53 of the sum of their magnitudes, n up to 402
    assert np.all(np.abs(val - ref.data) <= 402 * 2.0 ** -53 * mag.data)


def _product_is_right(A, B, terms):
    """Structure, and sums of up to `terms` products in any order: terms * 2^-53 of the sum of their magnitudes."""
    C = dev.spgemm(_device(A), _device(B))
    pos, crd, val = C.pos.cpu().numpy(), C.crd.cpu().numpy(), C.val.cpu().numpy()
    ref, mag = A @ B, abs(A) @ abs(B)
    ref.sort_indices(), mag.sort_indices()
    assert np.array_equal(pos, mag.indptr) and np.array_equal(crd, mag.indices) and np.array_equal(crd, ref.indices)
    assert np.all(np.abs(val - ref.data) <= terms * 2.0 ** -53 * mag.data)


def test_more_long_rows_than_there_is_memory_for():
    """128 MB hold the bitmaps of 1310 rows of B in 819,200 columns that are stored; the others are walked like short rows."""
    rng = np.random.default_rng(5)
    stored = (np.arange(819200) * 1.7).astype(np.int64)                   # of 1,400,000 columns
    lens = [819200, 3200, 3199] + [3300] * 1400 + [40] * 300
    brows = [stored] + [np.sort(stored[rng.choice(819200, n, replace=False)]) for n in lens[1:]]
    B = _csr(brows, rng.uniform(0.5, 1, sum(lens)), (len(brows), 1400000))
    arows = [np.array([0])] + [np.sort(rng.choice(np.arange(1, len(brows)), 4, replace=False)) for _ in range(3300)]
    A = _csr(arows, rng.uniform(-1, 1, sum(map(len, arows))), (len(arows), len(brows)))
    assert np.count_nonzero(np.diff(B.indptr) >= 3200) > 1310 and A.shape[0] * 175000 > 64 * B.nnz
    _product_is_right(A, B, 4)


def test_long_rows_in_columns_that_keep_their_numbers():
    """All columns stored, and five products per word of the bitmaps."""
    rng = np.random.default_rng(6)
    lens = [511, 512, 513] + [2000] * 700 + [30] * 100
    brows = [np.sort(rng.choice(100000, n, replace=False)) for n in lens]
    B = _csr(brows, rng.uniform(0.5, 1, sum(lens)), (len(brows), 100000))
    arows = [np.array([0]), np.array([1, 2]), np.arange(len(brows))] + [np.sort(rng.choice(len(brows), 10, replace=False)) for _ in range(8000)]
    A = _csr(arows, rng.uniform(-1, 1, sum(map(len, arows))), (len(arows), len(brows)))
    assert np.diff(B.indptr)[A.indices].sum() > 4 * A.shape[0] * 3125 and A.shape[0] * 12500 > 64 * B.nnz
    _product_is_right(A, B, len(brows))
