"""Calls on a batch handle outside a solve, with members that were done in the
solve before: the product and the preconditioner of all members' rows."""
import numpy as np
import pytest

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ensemble import EnsembleLinear
from modflow6_gb300.ims import ImsLinearSettings
from test_gpu_batch_products import grid

pytestmark = pytest.mark.gpu

SHAPES = [(1, 20, 30), (2, 9, 40), (1, 1, 7)]


@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("shapes", [None, SHAPES], ids=["general", "grids"])
def test_product_and_preconditioner_after_a_solve(gblib, shapes, precision):
    rng = np.random.default_rng(2)
    ia, ja, am, mrow = [np.zeros(1, np.int64)], [], [], [0]
    for s in SHAPES:
        i, j, a = grid(*s, rng)
        ja.append(j + mrow[-1])
        ia.append(i[1:] + ia[-1][-1])
        am.append(a)
        mrow.append(mrow[-1] + i.size - 1)
    ia, ja = np.concatenate(ia).astype(np.int32), np.concatenate(ja).astype(np.int32)
    am, n = np.concatenate(am), mrow[-1]
    v = rng.standard_normal(n)
    ens = EnsembleLinear(ImsLinearSettings(dvclose=1e-9, rclose=1e-8, iter1=200, precision=precision)
                         ).allocate(np.array(mrow, np.int32), ia, ja, shapes)
    assert gblib.gbims_factor(ens._h, _lib.dptr(am), None) == 0
    want = np.zeros(n)
    rows = np.repeat(np.arange(n), np.diff(ia))
    np.add.at(want, rows, am * v[ja])
    scale = np.zeros(n)
    np.add.at(scale, rows, np.abs(am * v[ja]))
    apc = np.zeros(ja.size)
    assert gblib.gbims_get_apc(ens._h, _lib.dptr(apc)) == 0
    o = oracle.Ims(oracle.settings(), ia, ja)
    zo = oracle.ilu0a(apc, o.iapc(), o.japc(), v, fma=True)
    # the FP32 and df64 forms of the sweeps, relative to the result's scale: two
    # sweeps of up to 70 levels, 8 roundings a row that nothing damps, are
    # 7e-5 in FP32 and 2e-12 at df64's 2^-48
    tol = 1e-3 if precision == _lib.GBIMS_MIXED else 1e-10
    for solves in range(2):  # before the first solve, and after one
        y, z = np.full(n, np.nan), np.full(n, np.nan)
        assert gblib.gbims_matvec(ens._h, _lib.dptr(v), _lib.dptr(y)) == 0
        # at most 7 products and 6 sums, in FP64
        assert np.max(np.abs(y - want) / scale) <= 16 * 2.0 ** -53
        assert gblib.gbims_precondition(ens._h, _lib.dptr(v), _lib.dptr(z)) == 0
        assert np.max(np.abs(z - zo)) <= tol * np.max(np.abs(zo))
        if solves == 0:
            res = ens.apply(am.copy(), np.ones(n), np.zeros(n))
            assert all(r.icnvg == 1 for r in res)
    ens.close()
