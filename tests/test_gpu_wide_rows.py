"""ILUT factors whose band fills to the most entries a working row holds (256
a triangle) and one fewer, and wide levels of long rows: the application
against the oracle's, bit for bit, in FP64 and within an FP32 bound in the
mixed form."""
import numpy as np
import pytest

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ims import ImsLinear, ImsLinearSettings
from test_gpu_range import banded_pattern

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("columns", [255, 256])
def test_full_band_bitexact(gblib, columns, precision):
    n = 4 * columns
    ia, ja, amat = banded_pattern(n, [1, columns], seed=columns)
    ims = ImsLinear(ImsLinearSettings(ilinmeth=2, level=300, droptol=0.0, precision=precision)
                    ).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) == 0
    iapc, japc, apc, _ = oracle.ilut(ia, ja, amat, 300, 0.0)
    assert np.max(japc[:n] - iapc[:-1]) == columns == np.max(iapc[1:] - japc[:n])
    v = np.random.default_rng(1).standard_normal(n)
    zo = oracle.ilu0a(apc, iapc, japc, v, fma=True)
    z = np.zeros(n)
    for _ in range(2):
        assert gblib.gbims_precondition(ims._h, _lib.dptr(v), _lib.dptr(z)) == 0
        if precision == _lib.GBIMS_FP64:
            np.testing.assert_array_equal(z, zo)
        else:
            # a row adds up to 256 products (258 roundings of 6e-8 of the
            # result's scale); the factor's rows sum to about half, so the
            # errors of the rows before at most double it, in each sweep
            assert np.max(np.abs(z - zo)) <= 1e-4 * np.max(np.abs(zo))


def test_wide_levels_of_long_rows(gblib):
    """32 interleaved one-layer grids of 128 columns: levels of 32 rows of 128
    entries, whose slices are cut."""
    n = 8192
    ia, ja, amat = banded_pattern(n, [32, 32 * 128], seed=5)
    ims = ImsLinear(ImsLinearSettings(ilinmeth=2, level=150, droptol=0.0)).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) == 0
    iapc, japc, apc, _ = oracle.ilut(ia, ja, amat, 150, 0.0)
    assert np.max(japc[:n] - iapc[:-1]) == 128
    v = np.random.default_rng(1).standard_normal(n)
    z = np.zeros(n)
    assert gblib.gbims_precondition(ims._h, _lib.dptr(v), _lib.dptr(z)) == 0
    np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, v, fma=True))
