"""The ILU0/MILU0 factor of full DIS grids (k_dia7_factor.cu) against the
oracle's, bit for bit: at the edges of blocks (32 lines), for single rows,
columns and layers, for pivots that fail or need the retries, for signed zeros
and for products of the dropped fill that overflow; a batch of grids against
the general batch."""
import math

import numpy as np
import pytest
import torch

import oracle
from modflow6_gb300 import _lib
from modflow6_gb300.ensemble import EnsembleLinear
from modflow6_gb300.ims import ImsLinear, ImsLinearSettings
from test_gpu_batch_products import SHAPES, grid

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (1, 1, 40), (1, 40, 1), (40, 1, 1), (2, 2, 2), (1, 31, 5), (3, 32, 17), (2, 33, 3),
         (3, 65, 31), (4, 64, 2), (1, 20, 30), (5, 90, 90)]


def factor(gblib, ims, amat, nja):
    apc = np.zeros(nja)
    assert gblib.gbims_factor(ims._h, _lib.dptr(amat), None) >= 0
    assert gblib.gbims_get_apc(ims._h, _lib.dptr(apc)) == 0
    return apc


def change(kind, amat, ia):
    a = amat.copy()
    n = ia.size - 1
    rng = np.random.default_rng(7)
    if kind == "pivot":  # diagonals of the other sign and zero: retries
        a[ia[:-1][rng.uniform(size=n) < 0.05]] *= -0.001
        a[ia[n // 2]] = 0.0
    elif kind == "zeros":
        off = np.setdiff1d(np.arange(a.size), ia[:-1])
        a[off[rng.uniform(size=off.size) < 0.3]] = -0.0
    elif kind == "overflow":  # both sides of a dropped product near the limit
        a *= 2.0 ** (rng.integers(-3, 4, a.size) * 300)
    return a


def restated(ia, ja, amat, relax, nan_sign):
    """ims_base_pcilu0 with ims_base_pcu's retries (ImsLinearBase.f90:761-864,
    :928-1042), the sign of a NaN pivot given: the pivot test reads it, and
    which sign an invalid operation has is the processor's choice."""
    n = ia.size - 1
    rows = [sorted((int(ja[k]), float(amat[k])) for k in range(ia[r], ia[r + 1])) for r in range(n)]
    diag, off = [0.0] * n, [{c: 0.0 for c, _ in row if c != r} for r, row in enumerate(rows)]
    flag, delta, count = 0, 0.0, 0
    while True:
        failed = False
        for r in range(n):
            w = {c: 0.0 + v for c, v in rows[r]}
            rs = 0.0
            for c in [c for c in w if c < r]:
                w[c] = tl = w[c] * diag[c]
                for u, v in off[c].items():
                    if u > c and u in w:
                        w[u] -= tl * v
                    elif u > c:
                        rs += tl * v
            d = w.pop(r)
            tl = (1.0 + delta) * d - relax * rs
            if math.copysign(d, tl if tl == tl else nan_sign) != d or tl == 0.0:
                if flag <= 1:
                    failed = True
                    break
                tl = math.copysign(1.0e-6, d)
            diag[r], off[r] = 1.0 / tl, w
        if not failed or count == 10:
            break
        delta, flag, count = 1.5 * delta + 1.0e-3, 0, count + 1
        if delta > 0.5:
            delta, flag = 0.5, 2
    return np.array(diag + [v for w in off for v in w.values()])


@pytest.mark.parametrize("kind", ["plain", "pivot", "zeros", "overflow"])
@pytest.mark.parametrize("relax", [0.0, 0.97])
@pytest.mark.parametrize("shape", GRIDS, ids=str)
def test_wave_factor_bitexact(gblib, shape, relax, kind):
    ia, ja, am = grid(*shape, np.random.default_rng(sum(shape)))
    ia, ja = ia.astype(np.int32), ja.astype(np.int32)
    am = change(kind, am, ia)
    n = ia.size - 1
    o = oracle.Ims(oracle.settings(relax=relax), ia, ja)
    o.apply(am.copy(), np.ones(n), np.zeros(n))
    want = o.apc()
    if kind == "overflow":
        one = torch.ones(1, dtype=torch.float64, device="cuda")
        sign = -1.0 if bool(torch.signbit(one - 0.0 * (one * np.inf))) else 1.0
        want = restated(ia, ja, am, relax, sign)
    ims = ImsLinear(ImsLinearSettings(structure=shape, relax=relax)).imslinear_allocate(n, ia, ja)
    for _ in range(2):
        apc = factor(gblib, ims, am, ja.size)
        nan = np.isnan(want)
        np.testing.assert_array_equal(np.isnan(apc), nan)
        np.testing.assert_array_equal(apc.view(np.uint64)[~nan], want.view(np.uint64)[~nan])


@pytest.mark.parametrize("relax", [0.0, 0.97])
def test_wave_factor_batch(gblib, relax):
    rng = np.random.default_rng(4)
    ia, ja, am, mrow = [np.zeros(1, np.int64)], [], [], [0]
    for s in SHAPES:
        i, j, a = grid(*s, rng)
        ja.append(j + mrow[-1])
        ia.append(i[1:] + ia[-1][-1])
        am.append(a)
        mrow.append(mrow[-1] + i.size - 1)
    ia, ja = np.concatenate(ia).astype(np.int32), np.concatenate(ja).astype(np.int32)
    am, mrow = np.concatenate(am), np.array(mrow, np.int32)
    out = []
    for sh in (None, SHAPES):
        ens = EnsembleLinear(ImsLinearSettings(relax=relax)).allocate(mrow, ia, ja, sh)
        out.append(factor(gblib, ens, am, ja.size))
        ens.close()
    np.testing.assert_array_equal(out[0], out[1])
