"""The count of one triangular matrix with itself, in another order of its vertices: graphs with and without vertices beyond the hub columns,
upper triangles, and matrices that have to be counted as they are."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from comet_b200 import device as dev  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _graph(kind, n, m, seed):
    """Edges (i > j) with hubs, or without any."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rand = lambda k: torch.rand(k, generator=gen, device="cuda", dtype=torch.float64)
    p, q = (1, 1) if kind == "even" else (4, 2)
    i, j = (n * rand(m) ** p).long(), (n * rand(m) ** q).long()
    if kind == "star":                           # a vertex next to all, a clique, and 200 vertices next to all of the clique
        c = n // 2 + torch.arange(300, device="cuda")
        other = torch.cat([c, (n * rand(200)).long()])
        i = torch.cat([i, torch.arange(n, device="cuda"), c.repeat_interleave(500)])
        j = torch.cat([j, torch.zeros(n, dtype=torch.int64, device="cuda"), other.repeat(300)])
    perm = torch.randperm(n, generator=gen, device="cuda")
    i, j = perm[i], perm[j]
    key = torch.unique(torch.maximum(i, j) * n + torch.minimum(i, j))
    i, j = torch.div(key, n, rounding_mode="floor"), key % n
    return i[i != j], j[i != j]


def _device(rows, cols, n):
    key = torch.sort(rows * n + cols)[0]
    rows, cols = torch.div(key, n, rounding_mode="floor"), key % n
    pos = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    pos[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return dev.DeviceCSR(n, n, pos, cols, torch.ones(rows.numel(), dtype=torch.float64, device="cuda"))


def _by_blocks(D, cuts):
    """Blocks of rows are counted in the order they are stored in."""
    return sum(int(dev.masked_pair_count(D, D, D, a, b)) for a, b in zip(cuts[:-1], cuts[1:]))


@pytest.mark.parametrize("kind", ["skewed", "star", "even"])
@pytest.mark.parametrize("n,m", [(8000, 25000000), (16384, 15000000), (16500, 15000000), (300000, 8000000), (700000, 9000000)])
def test_graphs(kind, n, m):
    i, j = _graph(kind, n, m, n)
    assert i.numel() >= max(6000000, 10 * n)
    L, U = _device(i, j, n), _device(j, i, n)
    want = _by_blocks(L, [0, n // 2, n])
    assert want > 0
    assert int(dev.masked_pair_count(L, L, L)) == want
    assert int(dev.masked_pair_count(U, U, U)) == want
    assert int(dev.masked_pair_count(L, L, L)) == want


@pytest.mark.parametrize("what", ["both triangles", "diagonal", "repeats", "one entry above"])
def test_matrices_that_keep_their_order(what):
    n = 60000
    i, j = _graph("skewed", n, 8000000, 8)
    also = lambda v, *k: torch.cat([v, torch.tensor(k, device="cuda")])
    if what == "both triangles":
        i, j = torch.cat([i, j]), torch.cat([j, i])
    elif what == "diagonal":
        i, j = also(i, 77), also(j, 77)
    elif what == "repeats":
        i, j = torch.cat([i, i[1000:1003]]), torch.cat([j, j[1000:1003]])
    else:
        i, j = also(i, 3), also(j, n - 1)
    D = _device(i, j, n)
    assert D.nnz >= max(6000000, 10 * n)
    assert int(dev.masked_pair_count(D, D, D)) == _by_blocks(D, [0, n // 3, n])


def test_against_the_oracle():
    n = 20000
    i, j = _graph("skewed", n, 14000000, 1)
    D = _device(i, j, n)
    pos, crd = D.pos.cpu().numpy(), D.crd.cpu().numpy()
    L = oracle.SparseArrays("CSR", n, n, np.array([n]), np.array([-1]), pos, crd, np.ones(crd.size))
    assert D.nnz >= 6000000
    assert int(dev.masked_pair_count(D, D, D)) == oracle.masked_pair_count_rowparallel(L, L, L)


@pytest.mark.parametrize("hub", [0, 1])
def test_a_column_at_the_same_place_of_every_row(hub):
    """Rows of an even number of entries that all end in the last column, and rows of one length that lies in one bucket of degrees."""
    n = 400000
    i, j = _graph("skewed", n, 9000000, 11)
    i, j = j, i                                          # rows are the lower numbers
    keep = j != n - 1
    i, j = i[keep], j[keep]
    if hub:
        order = torch.argsort(i * n + j)
        i, j = i[order], j[order]
        count = torch.bincount(i, minlength=n)
        first = torch.cumsum(count, 0) - count
        drop = first[(count % 2 == 0) & (count > 0)]     # one entry less where the number is even
        keep = torch.ones(i.numel(), dtype=torch.bool, device="cuda")
        keep[drop] = False
        i, j = i[keep], j[keep]
        rows = torch.nonzero(torch.bincount(i, minlength=n)).flatten()
        i, j = torch.cat([i, rows]), torch.cat([j, torch.full_like(rows, n - 1)])
    else:
        rows = torch.arange(n - 20, device="cuda").repeat_interleave(16)
        i, j = rows, rows + 1 + torch.arange(16, device="cuda").repeat(n - 20)
    D = _device(i, j, n)
    assert D.nnz >= max(6000000, 10 * n)
    assert int(dev.masked_pair_count(D, D, D)) == _by_blocks(D, [0, n // 3, n])


def test_more_rows_than_there_is_memory_for():
    """Rows of 64 and more entries in the hub columns, twice as many as there is room for bitmaps of."""
    n, m = 110000, 128
    gen = torch.Generator(device="cuda")
    gen.manual_seed(12)
    i = torch.arange(n, device="cuda").repeat_interleave(m)
    j = (torch.rand(n * m, generator=gen, device="cuda", dtype=torch.float64) * torch.where(torch.arange(n * m, device="cuda") % 16 == 0, n, 16000)).long()
    key = torch.unique(torch.maximum(i, j) * n + torch.minimum(i, j))
    i, j = torch.div(key, n, rounding_mode="floor"), key % n
    i, j = i[i != j], j[i != j]
    D = _device(i, j, n)
    rows = int((torch.bincount(i[j < 16000], minlength=n) >= 64).sum())
    assert D.nnz >= max(6000000, 10 * n) and (rows - 16384) * 512 > D.nnz * 2
    pos, crd = D.pos.cpu().numpy(), D.crd.cpu().numpy()
    L = oracle.SparseArrays("CSR", n, n, np.array([n]), np.array([-1]), pos, crd, np.ones(crd.size))
    assert int(dev.masked_pair_count(D, D, D)) == oracle.masked_pair_count_rowparallel(L, L, L)


def test_rows_that_do_not_ascend():
    """Found out when the vertices have their new numbers already."""
    n = 60000
    i, j = _graph("skewed", n, 8000000, 8)
    D = _device(i, j, n)
    want = int(dev.masked_pair_count(D, D, D))
    p = int(D.pos[torch.diff(D.pos).argmax()])
    D.crd[p + 1:p + 3] = D.crd[p + 1:p + 3].flip(0)
    assert D.nnz >= max(6000000, 10 * n)
    assert int(dev.masked_pair_count(D, D, D)) == want
