"""Rows whose number of products lies at the bins' limits: few and many columns, long and short rows of B, empty rows, both
folds, repeated columns."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402

pytestmark = pytest.mark.gpu


def _pair(ncols, kind):
    """A row for each number of products: with B's rows of one entry or of up to 97, or one long row of B."""
    rng = np.random.default_rng(7)
    wanted = [0, 1, 255, 256, 257, 300, 511, 512, 700, 1023, 1024, 1025, 1500]
    lens = {"single": np.ones(1600, dtype=int), "mixed": rng.integers(0, 98, 400), "long": np.array([255, 256, 900, 1024, 1025, 1, 0])}[kind]
    brows = [np.sort(rng.integers(0, ncols, n)) for n in lens]
    B = sp.csr_matrix((rng.uniform(-1, 1, lens.sum()), np.concatenate(brows), np.concatenate([[0], np.cumsum(lens)])), shape=(lens.size, ncols))
    rows = []
    if kind == "long":
        rows = [np.array([i]) for i in range(lens.size)] + [np.array([5, 2]), np.array([6, 3]), np.array([0, 2])]
    else:
        for w in wanted:
            order = rng.permutation(lens.size)
            take = np.searchsorted(np.cumsum(lens[order]), w, side="right")
            rows.append(np.sort(order[:take]))
    A = sp.csr_matrix((rng.uniform(0.5, 1, sum(map(len, rows))), np.concatenate(rows), np.concatenate([[0], np.cumsum([len(x) for x in rows])])),
                      shape=(len(rows), lens.size))
    return A, B


def _device(m):
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return dev.DeviceCSR(*m.shape, up(m.indptr.astype(np.int64)), up(m.indices.astype(np.int64)), up(m.data))


@pytest.mark.parametrize("semiring", [api.PLUS_TIMES, api.MIN_PLUS])
@pytest.mark.parametrize("ncols", [1, 31, 2000, 128 * 32, 262144, 262145])
@pytest.mark.parametrize("kind", ["single", "mixed", "long"])
def test_rows_at_the_limits(kind, ncols, semiring):
    A, B = _pair(ncols, kind)
    dA, dB = _device(A), _device(B)
    C = dev.spgemm(dA, dB, semiring=semiring)
    pos, crd, val = C.pos.cpu().numpy(), C.crd.cpu().numpy(), C.val.cpu().numpy()
    for r in range(A.shape[0]):
        want = {}
        for k, a in zip(A.indices[A.indptr[r]:A.indptr[r + 1]], A.data[A.indptr[r]:A.indptr[r + 1]]):
            for j, b in zip(B.indices[B.indptr[k]:B.indptr[k + 1]], B.data[B.indptr[k]:B.indptr[k + 1]]):
                if semiring == api.PLUS_TIMES:
                    want[j] = want.get(j, 0.0) + a * b
                else:
                    want[j] = min(want.get(j, np.inf), a + b)
        keys = sorted(want)
        assert np.array_equal(crd[pos[r]:pos[r + 1]], keys)
        assert np.allclose(val[pos[r]:pos[r + 1]], [want[j] for j in keys], rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("ncols", [1070400, 1070401])      # the most columns whose bitmap fits the 257-to-1024 kernel, one more
def test_the_widest_matrices(ncols):
    test_rows_at_the_limits("mixed", ncols, api.PLUS_TIMES)
