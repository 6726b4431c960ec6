"""One symmetric matrix as both operands and mask: counted by halves.  Row lengths at the edges of the kernels, equal lengths, entries
on the diagonal, every semiring, and patterns with a single entry that has no mate."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _pattern(kind, n, rng):
    d = np.zeros((n, n), dtype=bool)
    if kind == "hubs":                       # rows around 128, 512 and 2048 entries among short ones
        for r, k in enumerate([1, 127, 128, 129, 511, 512, 513, 2047, 2048, 2049, n]):
            d[r, rng.choice(n, k, replace=False)] = True
        d |= rng.random((n, n)) < 0.004
    elif kind == "equal":                    # all rows alike
        d[(np.arange(n)[:, None] + np.arange(-40, 41)[None, :]) % n, np.arange(n)[:, None]] = True
    else:
        d = rng.random((n, n)) < 0.05
    d |= d.T
    if kind == "no diagonal":
        np.fill_diagonal(d, False)
    if kind == "one-sided":
        i, j = np.argwhere(np.triu(d, 1))[7]
        d[j, i] = False
    return d


@pytest.mark.parametrize("kind,n,semirings", [("hubs", 2100, [api.PLUS_TIMES, api.PLUS_PAIR]), ("equal", 300, [api.PLUS_TIMES, api.PLUS_PAIR]),
                                              ("random", 200, range(8)), ("no diagonal", 333, [api.PLUS_TIMES, api.PLUS_PAIR]),
                                              ("one-sided", 200, range(8))])
def test_symmetric_patterns(kind, n, semirings):
    rng = np.random.default_rng(n)
    d = _pattern(kind, n, rng)
    pos = np.concatenate([[0], np.cumsum(d.sum(1))]).astype(np.int64)
    crd = np.nonzero(d)[1].astype(np.int64)
    aval, bval = rng.uniform(0.5, 1.5, crd.size), rng.uniform(0.5, 1.5, crd.size)
    up = lambda a: torch.from_numpy(a).cuda()
    p, c = up(pos), up(crd)
    A, B = dev.DeviceCSR(n, n, p, c, up(aval)), dev.DeviceCSR(n, n, p, c, up(bval))
    orc = lambda v: oracle.SparseArrays("CSR", n, n, np.array([n]), np.array([-1]), pos, crd, v)
    for semiring in semirings:
        C, ref = dev.spgemm(A, B, A, semiring), oracle.spgemm(orc(aval), orc(bval), orc(aval), semiring)
        assert np.array_equal(C.pos.cpu().numpy(), ref.a2pos) and np.array_equal(C.crd.cpu().numpy(), ref.a2crd)
        np.testing.assert_allclose(C.val.cpu().numpy(), ref.val, rtol=1e-12)
