"""The block sums (k_reduce.cuh): the order of the additions, bit for bit, at
the edges of warps and blocks and where another warp of the block adds (every
152 blocks); and the maxima's signs and rows, the smallest row among equals."""
import numpy as np
import pytest

from modflow6_gb300 import _lib
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings

pytestmark = pytest.mark.gpu

BLOCK = 256


def tree(v):
    """Block sums of v [blocks, 256]: lanes 16, 8, 4, 2, 1 apart, then warps."""
    for width in (32, 16, 8, 4, 2):
        v = v.reshape(*v.shape[:1], -1, width)
        v = v[..., :width // 2] + v[..., width // 2:]
    v = v.reshape(v.shape[0], BLOCK // 32)
    for width in (8, 4, 2):
        v = v[:, :width // 2] + v[:, width // 2:width]
    return v[:, 0]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 2053, 152 * 256 + 1, 700 * 256 - 3, 1216 * 256])
def test_sum_order(gblib, n):
    b = np.random.default_rng(n).standard_normal(n) * 10.0 ** np.random.default_rng(1).integers(-6, 7, n)
    pad = np.zeros(-(-n // BLOCK) * BLOCK)
    pad[:n] = b * b
    parts = tree(pad.reshape(-1, BLOCK))
    last = np.zeros(BLOCK)
    for i in range(0, parts.size, BLOCK):
        last[:parts[i:i + BLOCK].size] += parts[i:i + BLOCK]
    want = np.sqrt(tree(last[None, :])[0])
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1))
    ims.imslinear_allocate(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32))
    r = ims.imslinear_apply(-np.ones(n), b.copy(), np.zeros(n))
    assert r.summary["l2norm0"] == want


@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED])
@pytest.mark.parametrize("n", [1, 33, 257, 152 * 256 + 1, 400_000])
def test_largest_change(gblib, precision, n):
    # a diagonal system: the first step of PCG is the solution, +-3 in some
    # rows; of the rows with the largest step the smallest is reported
    rows = np.unique(np.array([n // 3, n // 2, n - 1]))
    b = np.full(n, 0.5)
    b[rows] = 3.0
    b[rows[0]] = -3.0
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1, precision=precision))
    ims.imslinear_allocate(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32))
    x = np.zeros(n)
    r = ims.imslinear_apply(np.ones(n), b.copy(), x)
    np.testing.assert_array_equal(x, b)
    assert r.summary["dvmax"] == -3.0
    assert r.summary["locdv"] == rows[0]
