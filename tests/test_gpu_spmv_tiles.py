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


def _boundaries(nnz):
    """Rows that end just before, on and behind the step up to which a row stays with the tile it starts in, rows that start on
    a boundary, and a row over more tiles than a warp has lanes."""
    lens, step = [], 0

    def row(n):
        nonlocal step
        lens.append(int(n))
        step += n + 1

    for behind in (0, 1, 2, 254, 255, 256, 257, 258, 2047, 2048, 2300, 2304, 2305, 6000):
        for start in (2047, 2048 - 17, 0, 1):
            row((start - 1 - step) % 2048)             # the next row starts `start` steps into a tile
            if start:
                row(2048 - step % 2048 + behind - 1)   # and ends `behind` steps behind a boundary
    row(80000)
    total = sum(lens)
    lens += [7] * ((nnz - total) // 7) + [(nnz - total) % 7]
    return np.array(lens)


@pytest.mark.parametrize("nnz", [310000, (1 << 20) - 1])
@pytest.mark.parametrize("kind", ["boundaries", "hubs", "middle", "one_row", "ragged"])
def test_sums_keep_their_order(kind, nnz):
    rng = np.random.default_rng(nnz)
    ncols = 9001
    if kind == "boundaries":
        lens = _boundaries(nnz)
    elif kind == "one_row":
        lens = np.array([0, nnz, 0])
    elif kind == "middle":                             # around the length from which a row is the tiles', cut and not
        lens = rng.integers(0, 1100, nnz // 400)
        lens = np.minimum(lens, np.maximum(nnz - np.concatenate([[0], np.cumsum(lens)[:-1]]), 0))
        lens[-1] += nnz - lens.sum()
    else:
        lens = np.diff(_matrix(kind, nnz).indptr)
    pos = np.concatenate([[0], np.cumsum(lens)])
    crd, val, x = rng.integers(0, ncols, nnz), rng.uniform(-1, 1, nnz), rng.uniform(-1, 1, ncols)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = dev.DeviceCSR(lens.size, ncols, up(pos), up(crd), up(val))
    y, y0 = dev.spmv(A, up(x)), rng.uniform(-1, 1, lens.size)
    added = dev.spmv(A, up(x), up(y0), accumulate=True)
    for _ in range(20):
        assert torch.equal(y, dev.spmv(A, up(x)))
        assert torch.equal(added, dev.spmv(A, up(x), up(y0), accumulate=True))
    # any order of a row's n terms is off by at most n 2^-53 of the sum of their sizes
    sums = lambda v: np.add.reduceat(np.concatenate([v, [0.0]]), np.minimum(pos[:-1], nnz)) * (lens > 0)
    ref, size = sums(val * x[crd]), sums(np.abs(val * x[crd]))
    assert np.all(np.abs(y.cpu().numpy() - ref) <= (lens + 1) * 2.0 ** -52 * size)
    assert np.all(np.abs(added.cpu().numpy() - ref - y0) <= (lens + 2) * 2.0 ** -52 * (size + np.abs(y0)))
    assert np.array_equal(dev.spmv(A, up(x), semiring=api.PLUS_PAIR).cpu().numpy(), lens)


def test_rows_behind_the_row_pointer_are_zero():
    """A row pointer shorter than the matrix: the rows it says nothing about are zero, whatever the new result's memory held."""
    n = 50000
    pos, crd = torch.arange(1001, device="cuda"), torch.arange(1000, device="cuda")
    A = dev.DeviceCSR(n, n, pos, crd, torch.ones(1000, device="cuda", dtype=torch.float64))
    x = torch.ones(n, device="cuda", dtype=torch.float64)
    dirty = torch.full((n,), 7.0, device="cuda", dtype=torch.float64)
    del dirty                                          # the allocator gives it out again
    y = dev.spmv(A, x)
    assert bool((y[:1000] == 1).all()) and not y[1000:].any()


@pytest.mark.parametrize("tiles,more", [(-1, 0), (-1, 1), (0, 0), (1024, 0), (1024, 1)])
def test_where_the_tiles_take_over(tiles, more):
    """As many tiles of 2048 steps (entries and row ends) as the chip has SMs, less one step; and the most that one launch
    takes, and one more."""
    steps = (tiles if tiles > 0 else torch.cuda.get_device_properties(0).multi_processor_count + tiles) * 2048 + more
    nnz = min(steps - 5000, 1000003)
    rng = np.random.default_rng(steps)
    pos = np.sort(np.concatenate([[0, nnz], rng.integers(0, nnz + 1, steps - nnz - 1)]))
    lens, crd, val, x = np.diff(pos), rng.integers(0, 9001, nnz), rng.uniform(-1, 1, nnz), rng.uniform(-1, 1, 9001)
    assert lens.size + nnz == steps
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = dev.DeviceCSR(lens.size, 9001, up(pos), up(crd), up(val))
    y = dev.spmv(A, up(x))
    assert all(torch.equal(y, dev.spmv(A, up(x))) for _ in range(3))
    ref, size = (np.bincount(np.repeat(np.arange(lens.size), lens), w, lens.size) for w in (val * x[crd], np.abs(val * x[crd])))
    assert np.all(np.abs(y.cpu().numpy() - ref) <= (lens + 1) * 2.0 ** -52 * size)
