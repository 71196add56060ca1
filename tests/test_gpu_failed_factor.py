"""A factorisation whose last retry still fails at a pivot: the rows before the
first failure hold that attempt's values, the others what they held (the
factor of the matrix before), bit for bit as in the oracle, run after run."""
import ctypes as C

import numpy as np
import pytest

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings

pytestmark = pytest.mark.gpu


def lines_pattern(offsets, seed, n=3000, line=50):
    """Lines of 50 rows, each row joined to the next of its line and to the
    rows `offsets` further on: a line's first row is eliminated long before the
    last rows of the lines before it."""
    rng = np.random.default_rng(seed)
    nb = [[] for _ in range(n)]
    for r in range(n):
        for q in [r + 1] * ((r + 1) % line != 0) + [r + o for o in offsets]:
            if q < n:
                nb[r].append(q)
                nb[q].append(r)
    ia, ja, a = np.zeros(n + 1, np.int32), [], []
    for r in range(n):
        row = sorted(nb[r])
        ja += [r] + row
        a += [-(len(row) + 1.0 + rng.uniform())] + list(rng.uniform(0.2, 1.0, len(row)))
        ia[r + 1] = len(ja)
    return ia, np.array(ja, np.int32), np.array(a)


@pytest.mark.parametrize("relax", [0.0, 0.97])
@pytest.mark.parametrize("rows", [[0], [2950], [1250, 2900, 1201], [31, 32], [2999]], ids=str)
@pytest.mark.parametrize("offsets", [[50], [50, 100, 150, 200, 250, 300]], ids=["short", "long"])
def test_rows_before_the_first_failure(gblib, offsets, rows, relax):
    ia, ja, good = lines_pattern(offsets, seed=4)
    n = ia.size - 1
    bad = good * np.random.default_rng(5).uniform(0.5, 1.5, good.size)
    for r in rows:  # a row without lower entries' values and a zero pivot, whatever delta
        k = np.arange(ia[r], ia[r + 1])
        bad[k[ja[k] <= r]] = 0.0
    o = oracle.Ims(oracle.settings(relax=relax, iter1=1), ia, ja)
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, relax=relax)).imslinear_allocate(n, ia, ja)
    apc, retries = np.zeros(ja.size), C.c_int()
    for amat in (good, bad, bad, good, bad):
        o.apply(amat.copy(), np.ones(n), np.zeros(n))
        assert gblib.gbims_factor(ims._h, _lib.dptr(amat), C.byref(retries)) >= 0
        assert retries.value == (11 if amat is bad else 0)
        assert gblib.gbims_get_apc(ims._h, _lib.dptr(apc)) == 0
        np.testing.assert_array_equal(apc, o.apc())
