"""SpMV where the kernels change: the sizes at which one launch, tiles and the chunk list take over, rows that end on tile
boundaries, span tiles or are empty, added values, plus-pair and stored rows only."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402

pytestmark = pytest.mark.gpu


def _matrix(kind, nnz, ncols=9001):
    rng = np.random.default_rng(3)
    if kind == "hubs":
        lens = np.minimum(rng.pareto(0.6, nnz // 8 + 1) * 2, ncols).astype(np.int64)
    elif kind == "tiles":          # 2047 entries and their row end fill a tile; then runs of empty rows
        lens = np.tile([2047, 2047, 5000, 0, 0, 2046, 1, 0] + [0] * 3000 + [3] * 50, nnz // 11000 + 1)
    else:
        lens = rng.integers(0, 33, nnz // 16 + 2)
    ends = np.minimum(np.cumsum(lens), nnz)
    ends[-1] = nnz
    pos = np.concatenate([[0], ends])
    return sp.csr_matrix((rng.uniform(-1, 1, nnz), rng.integers(0, ncols, nnz), pos), shape=(ends.size, ncols))


@pytest.mark.parametrize("nnz", [1, 50000, (1 << 18), (1 << 18) + 1, 300007, (1 << 20) - 1, (1 << 20), 1200000, (1 << 23), 9000000])
@pytest.mark.parametrize("kind", ["hubs", "tiles", "ragged"])
def test_sizes(kind, nnz):
    m = _matrix(kind, nnz)
    counts = np.diff(m.indptr)                         # scipy adds repeated entries up as it goes
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    arrays = [up(m.indptr.astype(np.int64)), up(m.indices.astype(np.int64)), up(m.data)]
    A, (n, ncols) = dev.DeviceCSR(*m.shape, *arrays), m.shape
    x = np.random.default_rng(nnz).uniform(-1, 1, ncols)
    ref, room = m @ x, 1e-13 * (abs(m) @ np.abs(x) + 1)
    assert np.all(np.abs(dev.spmv(A, up(x)).cpu().numpy() - ref) <= room)
    y = torch.ones(n, device="cuda", dtype=torch.float64)
    assert np.all(np.abs(dev.spmv(A, up(x), y, accumulate=True).cpu().numpy() - 1 - ref) <= 10 * room)
    assert np.array_equal(dev.spmv(A, up(x), semiring=api.PLUS_PAIR).cpu().numpy(), counts)
    ids = dev.DeviceCSR(2 * n, ncols, *arrays, row_ids=up(np.arange(n, dtype=np.int64) * 2 + 1))
    y = dev.spmv(ids, up(x)).cpu().numpy()
    assert np.all(np.abs(y[1::2] - ref) <= room) and not y[::2].any()
