"""Short rows counted with a bitmap of a warp's own: numbers of columns around words and the limit, products that all meet in a few
columns, up to 256 of them, and sums in the order of the sequential loop."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from comet_b200 import api  # noqa: E402
from comet_b200 import device as dev  # noqa: E402
from oracle import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _csr(rows, ncols, rng):
    pos = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return pos, np.concatenate(rows).astype(np.int64), rng.uniform(-1, 1, pos[-1])


@pytest.mark.parametrize("semirings", [[api.PLUS_TIMES], range(8)])
@pytest.mark.parametrize("ncols", [1, 32, 4096, 4097, 16384, 16385, 32767, 32768, 32769])
def test_short_rows(ncols, semirings):
    rng = np.random.default_rng(ncols)
    near = np.minimum(ncols - 1, np.array([0, 1, 31, 32, 63, 127, 128, 4095, 4096, ncols - 1]))
    brows = [np.sort(rng.integers(0, ncols, n)) for n in (0, 1, 2, 16, 31, 32, 33, 64, 127, 128, 255, 256)]
    brows += [np.sort(rng.choice(near, n)) for n in (3, 16, 40, 64)]                 # most of the products meet
    m = len(brows)
    arows = [[i] for i in range(m)] + [[12, 13, 14, 15], [15, 15, 15, 15], [3] * 16, [1] * 256, [12] * 85, [2, 1] * 40, [9, 9], []]
    arows += [rng.integers(1, 5, rng.integers(1, 17)) for _ in range(40)]
    A, B = _csr([np.sort(r) for r in arows], m, rng), _csr(brows, ncols, rng)
    up = lambda a: torch.from_numpy(a).cuda()
    dA, dB = dev.DeviceCSR(len(arows), m, *map(up, A)), dev.DeviceCSR(m, ncols, *map(up, B))
    orc = lambda t, nr, nc: oracle.SparseArrays("CSR", nr, nc, np.array([nr]), np.array([-1]), *t)
    for semiring in semirings:
        C, ref = dev.spgemm(dA, dB, semiring=semiring), oracle.spgemm(orc(A, len(arows), m), orc(B, m, ncols), None, semiring)
        assert np.array_equal(C.pos.cpu().numpy(), ref.a2pos) and np.array_equal(C.crd.cpu().numpy(), ref.a2crd)
        short = np.repeat(np.array([sum(len(brows[k]) for k in r) <= 256 for r in arows]), np.diff(ref.a2pos))
        assert np.array_equal(C.val.cpu().numpy()[short], ref.val[short])
        np.testing.assert_allclose(C.val.cpu().numpy(), ref.val, rtol=1e-12, atol=1e-13)
