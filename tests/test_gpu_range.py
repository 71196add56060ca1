"""The range sweeps of general patterns (k_range.cu) against the oracle's
ilu0a, bit for bit in FP64: at the edges of slices (32 rows) and ranges (2048
rows), for rows from no to 40 lower entries, dependencies inside a range, on
the range before and far back, and non-finite right-hand sides."""
import numpy as np
import pytest

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings

pytestmark = pytest.mark.gpu


def banded_pattern(n, offsets, seed, keep=1.0):
    """A symmetric pattern with the given band offsets, each pair kept with
    probability `keep`; diagonal first, the rest ascending."""
    rng = np.random.default_rng(seed)
    nb = [[] for _ in range(n)]
    for o in offsets:
        for r in np.flatnonzero(rng.uniform(size=max(0, n - o)) < keep):
            nb[r].append(r + o)
            nb[r + o].append(r)
    ia = np.zeros(n + 1, np.int32)
    ja, a = [], []
    for r in range(n):
        row = sorted(set(nb[r]))
        ja += [r] + row
        a += [-(len(row) + 1.0 + rng.uniform())] + list(rng.uniform(0.2, 1.0, len(row)))
        ia[r + 1] = len(ja)
    return ia, np.array(ja, np.int32), np.array(a)


CASES = {
    "1": (1, [], 1.0), "31-diagonal": (31, [], 1.0), "33-chain": (33, [1], 1.0),
    "2047": (2047, [1, 45], 1.0), "2048": (2048, [1, 45], 1.0), "2049": (2049, [1, 45], 1.0),
    "4100-far": (4100, [1, 50, 2500], 1.0), "6200-ragged": (6200, [1, 7, 60, 61, 62, 2100, 4000], 0.6),
    "2300-wide": (2300, list(range(1, 21)) + list(range(2000, 2020)), 0.9),
    "700-short-and-long": (700, [1] + list(range(300, 330)), 0.5),
}


@pytest.mark.parametrize("name", CASES)
def test_range_sweeps_bitexact(gblib, name):
    n, offsets, keep = CASES[name]
    ia, ja, amat = banded_pattern(n, offsets, seed=n, keep=keep)
    o = oracle.Ims(oracle.settings(), ia, ja)
    o.apply(amat.copy(), np.ones(n), np.zeros(n))
    rng = np.random.default_rng(1)
    v = rng.standard_normal(n)
    zo = oracle.ilu0a(o.apc(), o.iapc(), o.japc(), v, fma=True)
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL)).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) == 0
    z = np.zeros(n)
    for _ in range(3):  # successive launches, each with its own epoch
        z[:] = 0.0
        assert gblib.gbims_precondition(ims._h, _lib.dptr(v), _lib.dptr(z)) == 0
        np.testing.assert_array_equal(z, zo)
    # NaN (one with the payload that marks an empty slot) and infinity reach
    # the same rows as in the oracle
    w = v.copy()
    w[n // 3] = np.inf
    w.view(np.uint64)[n // 2] = 0x7FF8C0DE00000000
    wo = oracle.ilu0a(o.apc(), o.iapc(), o.japc(), w, fma=True)
    assert gblib.gbims_precondition(ims._h, _lib.dptr(w), _lib.dptr(z)) == 0
    np.testing.assert_array_equal(z, wo)  # NaN equal to NaN
    # the FP32 form, relative to the scale of the result: a row's error is at
    # most a few FP32 roundings per entry of the rows that feed it, and these
    # diagonally dominant factors damp them (1e-5 leaves more than 80 of them)
    m32 = ImsLinear(ImsLinearSettings(structure=GENERAL, precision=_lib.GBIMS_MIXED)
                    ).imslinear_allocate(n, ia, ja)
    assert gblib.gbims_factor(m32._h, _lib.dptr(amat), None) == 0
    assert gblib.gbims_precondition(m32._h, _lib.dptr(v), _lib.dptr(z)) == 0
    assert np.max(np.abs(z - zo)) <= 1e-5 * np.max(np.abs(zo))


@pytest.mark.parametrize("relax", [0.0, 0.97])
@pytest.mark.parametrize("name,n,offsets", [
    ("six", 700, [1, 2, 3, 30, 31, 32]), ("seven", 700, [1, 2, 3, 30, 31, 32, 33]),
    ("one-row", 1, []), ("chain", 200, [1]), ("wide-levels", 5000, [2500, 2501]),
    ("thirty", 400, list(range(1, 31)))])
def test_one_launch_factor_bitexact(gblib, name, n, offsets, relax):
    """The ILU0/MILU0 factor against the oracle's, bit for bit, at the edge
    between its short rows (six lower and upper entries) and long ones, for
    the narrowest and the widest levels, with and without the dropped fill."""
    ia, ja, amat = banded_pattern(n, offsets, seed=3 * n + len(offsets))
    o = oracle.Ims(oracle.settings(relax=relax), ia, ja)
    o.apply(amat.copy(), np.ones(n), np.zeros(n))
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, relax=relax)).imslinear_allocate(n, ia, ja)
    apc = np.zeros(ja.size)
    for _ in range(2):
        assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) >= 0
        assert gblib.gbims_get_apc(ims._h, _lib.dptr(apc)) == 0
        np.testing.assert_array_equal(apc, o.apc())
