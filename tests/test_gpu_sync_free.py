"""The sync-free sweeps of patterns with few levels (k_ilu.cu) against the oracle's
ilu0a, bit for bit in FP64: no entries, levels of one row and of many, rows of
many entries, more rows than threads, non-finite right-hand sides; between the
forms of the sweeps on one handle; and by several threads on handles of their
own."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings

pytestmark = pytest.mark.gpu


def random_pattern(n, degree, seed):
    """A random symmetric pattern of about `degree` pairs a row."""
    rng = np.random.default_rng(seed)
    p = np.unique(np.sort(rng.integers(0, n, (int(n * degree), 2)), 1), axis=0)
    p = p[p[:, 0] != p[:, 1]]
    r, c = np.concatenate([p[:, 0], p[:, 1]]), np.concatenate([p[:, 1], p[:, 0]])
    count = np.bincount(r, minlength=n)
    ia = np.concatenate([[0], np.cumsum(count + 1)]).astype(np.int32)
    rows = np.concatenate([np.arange(n), r])
    key = np.concatenate([np.full(n, -1), c])
    order = np.lexsort((key, rows))
    ja = np.concatenate([np.arange(n), c])[order].astype(np.int32)
    a = np.concatenate([-(count + 1.0 + rng.uniform(size=n)), rng.uniform(0.2, 1.0, r.size)])[order]
    return ia, ja, a


CASES = {"1": (1, 0), "31": (31, 0), "3000-diagonal": (3000, 0), "300-dense": (300, 12), "5000": (5000, 1),
         "40000": (40000, 3), "400000": (400000, 0.4)}


@pytest.mark.parametrize("name", CASES)
def test_sync_free_bitexact(gblib, name):
    n, degree = CASES[name]
    ia, ja, amat = random_pattern(n, degree, seed=n)
    o = oracle.Ims(oracle.settings(), ia, ja)
    o.apply(amat.copy(), np.ones(n), np.zeros(n))
    apc, iapc, japc = o.apc(), o.iapc(), o.japc()
    v = np.random.default_rng(1).standard_normal(n)
    zo = oracle.ilu0a(apc, iapc, japc, v, fma=True)
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL)).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) == 0
    z = np.zeros(n)

    def applied(rhs, want):
        for _ in range(3):  # successive launches, each with its own epoch
            z[:] = 0.0
            assert gblib.gbims_precondition(ims._h, _lib.dptr(rhs), _lib.dptr(z)) == 0
            np.testing.assert_array_equal(z, want)

    applied(v, zo)
    w = v.copy()
    w[n // 3] = np.inf
    w[n // 2] = np.nan
    applied(w, oracle.ilu0a(apc, iapc, japc, w, fma=True))  # NaN equal to NaN
    # launches per level and back, and whatever the tuner keeps: the words of one
    # form are not taken for the other's
    for mode in (0, 1):
        assert gblib.gbims_set_tuning(ims._h, -1, 0, mode) == 0
        applied(v, zo)
    assert gblib.gbims_autotune(ims._h, 2, C.byref(_lib.GbimsTuning())) == 0
    applied(v, zo)
    # the FP32 form: as in the range sweeps' test
    m32 = ImsLinear(ImsLinearSettings(structure=GENERAL, precision=_lib.GBIMS_MIXED)).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(m32._h, _lib.dptr(amat), None) == 0
    assert gblib.gbims_precondition(m32._h, _lib.dptr(v), _lib.dptr(z)) == 0
    assert np.max(np.abs(z - zo)) <= 1e-5 * np.max(np.abs(zo))


def test_side_by_side(gblib):
    """Sweeps of several handles at once, each with more blocks than its share of
    the GPU has places for: none waits for rows that nobody works on."""
    n = 400000
    ia, ja, amat = random_pattern(n, 0.4, seed=n)
    v = np.random.default_rng(2).standard_normal(n)
    lin = [ImsLinear(ImsLinearSettings(structure=GENERAL)).imslinear_allocate(n, ia, ja) for _ in range(3)]
    z = np.zeros((len(lin), n))
    for k, ims in enumerate(lin):
        assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) == 0
        assert gblib.gbims_precondition(ims._h, _lib.dptr(v), _lib.dptr(z[k])) == 0
    want, wrong = z[0].copy(), []
    assert np.array_equal(want, z[1])

    def run(k):
        times = _lib.GbimsKernelTimes()
        for _ in range(5):
            if gblib.gbims_time_kernels(lin[k]._h, 40, C.byref(times)) != 0:
                wrong.append(k)
            if gblib.gbims_precondition(lin[k]._h, _lib.dptr(v), _lib.dptr(z[k])) != 0 or not np.array_equal(z[k], want):
                wrong.append(k)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(lin))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong
