"""The inner loop as a graph (several iterations a body on small systems)
against the same iterations launched from the host: whole numbers and bits the
same wherever the loop ends within a body, by convergence or by the limit."""
import numpy as np
import pytest

from modflow6_gb300 import _lib
from modflow6_gb300.ims import ImsLinear, ImsLinearSettings

pytestmark = pytest.mark.gpu


def laplace(n):
    ia, ja, a = np.zeros(n + 1, np.int32), [], []
    for r in range(n):
        row = [c for c in (r - 1, r + 1, r - 40, r + 40) if 0 <= c < n]
        ja += [r] + row
        a += [-len(row) - 0.01] + [1.0] * len(row)
        ia[r + 1] = len(ja)
    return ia, np.array(ja, np.int32), np.array(a)


@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED])
@pytest.mark.parametrize("accel", [1, 2])
@pytest.mark.parametrize("limit", [1, 2, 3, 4, 5, 6, 500])
def test_graph_bodies_equal_host_loop(gblib, monkeypatch, precision, accel, limit):
    n = 1000
    ia, ja, amat = laplace(n)
    rhs = np.random.default_rng(3).standard_normal(n)
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("GBIMS_GRAPH", graph)
        ims = ImsLinear(ImsLinearSettings(ilinmeth=accel, iter1=limit, precision=precision))
        ims.imslinear_allocate(n, ia, ja)
        x = np.zeros(n)
        r = ims.imslinear_apply(amat.copy(), rhs.copy(), x)
        out.append((x, r.in_iter, r.icnvg))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1:] == out[1][1:]
    assert out[0][1] <= limit
