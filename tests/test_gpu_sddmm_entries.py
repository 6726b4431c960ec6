"""SDDMM over equal pieces of the entries: widths where lanes and vectors per lane change, even and odd, aligned and not, rows
that share batches, fill them, span pieces, and runs of empty rows longer than a window of row ends."""
import numpy as np
import pytest
import scipy.sparse as sp

torch = pytest.importorskip("torch")

from comet_b200 import device as dev  # noqa: E402

pytestmark = pytest.mark.gpu


def _matrix(kind, ncols=901):
    rng = np.random.default_rng(5)
    lens = {"short": rng.integers(0, 9, 1201), "long": np.array([700, 0, 33, 901, 1, 32, 31, 300]), "one": np.array([1]),
            "skewed": np.minimum(ncols, (rng.pareto(0.7, 800) * 2).astype(int)), "sparse": (rng.random(30000) < 0.01) * 3}[kind]
    lens = lens.astype(int)
    cols = np.concatenate([np.sort(rng.permutation(ncols)[:n]) for n in lens])
    return sp.csr_matrix((rng.uniform(-1, 1, cols.size), cols, np.concatenate([[0], np.cumsum(lens)])), shape=(lens.size, ncols))


def _check(m, X, Y):
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    A = dev.DeviceCSR(m.shape[0], m.shape[1], up(m.indptr.astype(np.int64)), up(m.indices.astype(np.int64)), up(m.data))
    got = dev.sddmm(A, X, Y).cpu().numpy()
    rows = np.repeat(np.arange(m.shape[0]), np.diff(m.indptr))
    x, y = X.cpu().numpy()[rows], Y.cpu().numpy()[m.indices]
    assert np.all(np.abs(got - m.data * (x * y).sum(1)) <= 1e-13 * (np.abs(x * y).sum(1) + 1))


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 24, 26, 33, 48, 64, 66, 97, 128, 129, 150, 201, 256, 258, 515])
@pytest.mark.parametrize("kind", ["short", "long", "skewed", "sparse", "one"])
def test_widths(kind, k):
    m = _matrix(kind)
    X, Y = (torch.rand((n, k), device="cuda", dtype=torch.float64) - 0.5 for n in m.shape)
    _check(m, X, Y)


@pytest.mark.parametrize("k", [2, 14, 64, 130])
def test_operands_that_only_allow_8_byte_accesses(k):
    m = _matrix("skewed")
    wide = torch.rand(m.shape[0] * k + 1, device="cuda", dtype=torch.float64)
    Y = torch.rand((m.shape[1], k), device="cuda", dtype=torch.float64)
    _check(m, wide[1:].view(m.shape[0], k), Y)
