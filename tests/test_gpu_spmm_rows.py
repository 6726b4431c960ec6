"""The kernels that SpMM picks by itself: matrices with and without long rows, at the widths where lanes, vectors per lane and
slices change, even and odd, aligned and not, stored, added and counted (plus-pair), all rows stored or some (DCSR)."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402

pytestmark = pytest.mark.gpu


def _matrix(kind, nrows=1531, ncols=777):
    rng = np.random.default_rng(11)
    lens = {"short": rng.integers(0, 13, nrows), "one_long": rng.integers(0, 4, nrows), "empty": np.zeros(nrows, dtype=int),
            "skewed": np.minimum(ncols, (rng.pareto(0.7, nrows) * 2).astype(int)), "one_row": np.array([ncols])}[kind]
    if kind == "one_long":
        lens[nrows // 2] = ncols
    cols = np.concatenate([np.sort(rng.permutation(ncols)[:n]) for n in lens]) if lens.sum() else np.zeros(0, dtype=int)
    pos = np.concatenate([[0], np.cumsum(lens)])
    return sp.csr_matrix((rng.uniform(-1, 1, cols.size), cols, pos), shape=(lens.size, ncols))


def _device(m, row_ids=None, nrows=None):
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ids = None if row_ids is None else up(row_ids.astype(np.int64))
    return dev.DeviceCSR(nrows or m.shape[0], m.shape[1], up(m.indptr.astype(np.int64)), up(m.indices.astype(np.int64)), up(m.data), ids)


def _same(C, m, ref, B):
    limit = 1e-13 * (abs(m) @ np.abs(B) + 1)
    assert np.all(np.abs(C.cpu().numpy() - ref) <= limit)


@pytest.mark.parametrize("k", [1, 2, 3, 5, 8, 9, 16, 18, 23, 24, 33, 49, 64, 65, 94, 96, 97, 129, 256, 258, 520, 1027])
@pytest.mark.parametrize("kind", ["short", "one_long", "skewed", "empty", "one_row"])
def test_widths(kind, k):
    m = _matrix(kind)
    rng = np.random.default_rng(k)
    B, C0 = rng.uniform(-1, 1, (m.shape[1], k)), rng.uniform(-1, 1, (m.shape[0], k))
    A, dB, ref = _device(m), torch.from_numpy(B).cuda(), m @ B
    _same(dev.spmm(A, dB), m, ref, B)
    _same(dev.spmm(A, dB, torch.from_numpy(C0).cuda(), accumulate=True), m, ref + C0, B)
    pairs = dev.spmm(A, dB, semiring=api.PLUS_PAIR).cpu().numpy()
    assert np.array_equal(pairs, np.repeat(np.diff(m.indptr)[:, None], k, axis=1))


@pytest.mark.parametrize("k", [4, 32, 80, 128])
@pytest.mark.parametrize("kind", ["short", "skewed"])
def test_operands_that_only_allow_8_byte_accesses(kind, k):
    m = _matrix(kind)
    wide = torch.rand((m.shape[1], k + 3), device="cuda", dtype=torch.float64)
    B = wide[:, 1:k + 1]                               # odd row stride and an address 8 bytes off
    _same(dev.spmm(_device(m), B), m, m @ B.cpu().numpy(), B.cpu().numpy())


@pytest.mark.parametrize("k", [6, 41, 70, 128])
@pytest.mark.parametrize("kind", ["short", "one_long", "skewed"])
def test_stored_rows_only(kind, k):
    m = _matrix(kind)
    ids = np.arange(m.shape[0]) * 3 + 1
    B = np.random.default_rng(k).uniform(-1, 1, (m.shape[1], k))
    C = dev.spmm(_device(m, ids, 3 * m.shape[0] + 1), torch.from_numpy(B).cuda())
    _same(C[1::3], m, m @ B, B)
    assert not C[0::3].any() and not C[2::3].any()


@pytest.mark.parametrize("k", [1, 6, 33, 64, 200, 600])
def test_small_products_are_the_same_to_the_bit(k):
    m = _matrix("skewed")
    A, B = _device(m), torch.rand((m.shape[1], k), device="cuda", dtype=torch.float64)
    C = dev.spmm(A, B)
    assert all(torch.equal(C, dev.spmm(A, B)) for _ in range(5))
    if k > 6:                      # and a panel's sums are those of the whole product
        assert torch.equal(C[:, :6], dev.spmm(A, B[:, :6]))


def _hubs(nnz):
    """Short rows, and among them rows of one piece up to more units of pieces than a warp adds up alone."""
    rng = np.random.default_rng(nnz)
    hubs = [31, 33, 255, 257, 991, 1023, 1025, 1057, 8190, 8500, 16000, 17000, 39999]
    lens = rng.integers(0, 9, (nnz - sum(hubs)) // 4)
    lens[rng.permutation(lens.size)[:len(hubs)]] = hubs
    cols = rng.integers(0, 5000, lens.sum())
    pos = np.concatenate([[0], np.cumsum(lens)])
    return sp.csr_matrix((rng.uniform(-1, 1, cols.size), cols, pos), shape=(lens.size, 5000))


@pytest.mark.parametrize("k", [1, 4, 7, 17, 33, 48, 62, 65, 129, 201])
@pytest.mark.parametrize("nnz", [100000, 900000])
def test_sums_keep_their_order(nnz, k):
    """Rows cut into pieces: every call adds in the same order, below 64 columns and for every odd width."""
    m = _hubs(nnz)
    lens = np.diff(m.indptr)[:, None]
    rng = np.random.default_rng(k)
    B, C0 = rng.uniform(-1, 1, (m.shape[1], k)), rng.uniform(-1, 1, (m.shape[0], k))
    A, dB, dC = _device(m), torch.from_numpy(B).cuda(), torch.from_numpy(C0).cuda()
    C, acc = dev.spmm(A, dB), dev.spmm(A, dB, dC.clone(), accumulate=True)
    for _ in range(4):
        assert torch.equal(C, dev.spmm(A, dB))
        assert torch.equal(acc, dev.spmm(A, dB, dC.clone(), accumulate=True))
    # either order of a row's n + 1 terms is off by at most (n + 1) 2^-53 of the sum of their sizes
    n, size = lens + 1.0, sp.csr_matrix((np.abs(m.data), m.indices, m.indptr), shape=m.shape) @ np.abs(B)
    assert np.all(np.abs(C.cpu().numpy() - m @ B) <= n * 2.0 ** -52 * size)
    assert np.all(np.abs(acc.cpu().numpy() - (m @ B + C0)) <= (n + 1) * 2.0 ** -52 * (size + np.abs(C0)))
    dC = torch.from_numpy(C0).cuda()
    pairs = dev.spmm(A, dB, dC.clone(), semiring=api.PLUS_PAIR, accumulate=True)
    assert torch.equal(pairs, torch.from_numpy(C0 + lens).cuda())
