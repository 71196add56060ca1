"""A tuned solve of a system with fused products against the untuned one, bit for
bit: the tuner changes no cell's arithmetic and no order of a sum."""
import ctypes as C

import numpy as np
import pytest

from modflow6_gb300 import _lib
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings
from test_gpu_batch_products import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accel", [1, 2])
@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("general", [False, True], ids=["dis", "general"])
def test_tuned_solve_is_the_untuned_one(gblib, general, precision, accel):
    shape = (3, 150, 140)
    ia, ja, amat = grid(*shape, np.random.default_rng(6))
    ia, ja, n = ia.astype(np.int32), ja.astype(np.int32), ia.size - 1
    rhs = np.random.default_rng(7).standard_normal(n)
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL if general else shape, ilinmeth=accel, iter1=400,
                                      dvclose=1e-8, rclose=1e-6, precision=precision)).imslinear_allocate(n, ia, ja)
    out = []
    for tuned in range(3):
        x = np.zeros(n)
        r = ims.imslinear_apply(amat.copy(), rhs.copy(), x)
        out.append((x, r.in_iter, r.icnvg))
        t = _lib.GbimsTuning()
        assert gblib.gbims_autotune(ims._h, 5, C.byref(t)) == 0
        assert t.reduction_blocks == (n + 255) // 256
    assert out[0][2] == 1
    for x, it, cnvg in out[1:]:
        np.testing.assert_array_equal(x, out[0][0])
        assert (it, cnvg) == out[0][1:]
