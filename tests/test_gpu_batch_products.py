"""The index-free products of a batch of full DIS grids against the general
ones of the same batch, bit for bit: members of less than a block, of whole
chunks (2048 rows) and one row more, single rows, columns and layers."""
import numpy as np
import pytest

from modflow6_gb300 import _lib
from modflow6_gb300.ensemble import EnsembleLinear
from modflow6_gb300.ims import ImsLinearSettings

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 5), (5, 1, 1), (1, 20, 30), (2, 32, 32), (1, 1, 2049), (3, 32, 64), (4, 7, 300)]


def grid(nlay, nrow, ncol, rng):
    """CSR of a symmetric 7-point matrix, diagonal first."""
    n = nlay * nrow * ncol
    node = np.arange(n).reshape(nlay, nrow, ncol)
    nb = [[] for _ in range(n)]
    for axis in (0, 1, 2):
        a = np.take(node, range(node.shape[axis] - 1), axis).ravel()
        b = np.take(node, range(1, node.shape[axis]), axis).ravel()
        for p, q, c in zip(a, b, rng.uniform(0.1, 2.0, a.size)):
            nb[p].append((q, c))
            nb[q].append((p, c))
    ia, ja, am = [0], [], []
    for r in range(n):
        row = sorted(nb[r])
        ja += [r] + [q for q, _ in row]
        am += [-sum(c for _, c in row) - 0.05] + [c for _, c in row]
        ia.append(len(ja))
    return np.array(ia), np.array(ja), np.array(am)


@pytest.mark.parametrize("shapes", [SHAPES[:1], SHAPES[4:5], SHAPES])
def test_batch_products_bitexact(gblib, shapes):
    rng = np.random.default_rng(len(shapes))
    ia, ja, am, mrow = [np.zeros(1, np.int64)], [], [], [0]
    for s in shapes:
        i, j, a = grid(*s, rng)
        ja.append(j + mrow[-1])
        ia.append(i[1:] + ia[-1][-1])
        am.append(a)
        mrow.append(mrow[-1] + i.size - 1)
    ia, ja = np.concatenate(ia).astype(np.int32), np.concatenate(ja).astype(np.int32)
    am, mrow = np.concatenate(am), np.array(mrow, np.int32)
    rhs = rng.standard_normal(mrow[-1])
    x0 = rng.standard_normal(mrow[-1])
    out = []
    for sh in (None, shapes):
        ens = EnsembleLinear(ImsLinearSettings(dvclose=1e-9, rclose=1e-8, iter1=200)).allocate(mrow, ia, ja, sh)
        y = np.zeros(x0.size)
        assert gblib.gbims_factor(ens._h, _lib.dptr(am), None) == 0
        assert gblib.gbims_matvec(ens._h, _lib.dptr(x0), _lib.dptr(y)) == 0
        res = ens.apply(am.copy(), rhs.copy(), x0.copy())  # the residual's norm per member
        out.append((y, [r.summary["l2norm0"] for r in res]))
        ens.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
