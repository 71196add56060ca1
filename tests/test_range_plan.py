"""The plans of the range sweeps (k_range.cu), walked on the host as the kernel
walks them, against the oracle's ilu0a, bit for bit: every range size of the
tuner and the smallest, patterns of no to 256 entries a triangle (the most an
ILUT row keeps), and rows whose slice is as wide as its header can say."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle

ROOT = Path(__file__).resolve().parents[1]
INFO = ("R", "ranges", "stages", "maxblock", "slices")


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("range_plan") / "range_plan.so"
    abi = ROOT / "tests" / "c_abi"
    cmd = ["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
           "-Xcompiler", "-ffp-contract=off", "--expt-relaxed-constexpr", "-I",
           str(ROOT / "modflow6_gb300" / "csrc"), "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic",
           str(abi / "range_plan.cu"), str(abi / "host_cudart.cpp"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(str(out))


def factor_pattern(n, lower, seed):
    """IAPC/JAPC/APC of a factor whose row r has the lower entries lower(r),
    its transpose above; the pivots first, as in ILU0's storage."""
    rng = np.random.default_rng(seed)
    low = [sorted(c for c in lower(r) if 0 <= c < r) for r in range(n)]
    up = [[] for _ in range(n)]
    for r, cs in enumerate(low):
        for c in cs:
            up[c].append(r)
    iapc, japc = np.zeros(n + 1, np.int32), [0] * n
    iapc[0] = n
    for r in range(n):
        japc += low[r]
        japc[r] = len(japc)
        japc += up[r]
        iapc[r + 1] = len(japc)
    japc = np.array(japc, np.int32)
    wide = max(1, max(len(c) for c in low))
    apc = rng.uniform(-1.0, 1.0, japc.size) / wide
    apc[:n] = rng.uniform(0.5, 2.0, n)
    return iapc, japc, apc


def walk(plans, iapc, japc, apc, v, rows, fp32=False):
    """Both sweeps over the plans; the result and what the plans look like."""
    t = np.float32 if fp32 else np.float64
    fn = plans.range_walk32 if fp32 else plans.range_walk64
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    n = iapc.size - 1
    a, rhs, infos = apc.astype(t), v.astype(t), []
    for forward in (1, 0):
        out, info = np.full(n, np.nan, t), np.zeros(5, np.int32)
        rc = fn(n, p(iapc), p(japc), japc.size, p(a), forward, rows, p(rhs), p(out), p(info))
        assert rc == 0, (rc, forward, info)
        infos.append(dict(zip(INFO, info)))
        rhs = out
    return rhs, infos


def band(w):
    return lambda r: range(r - w, r)


PATTERNS = {
    "diagonal": (40, lambda r: []), "chain": (100, band(1)),
    "grid": (9000, lambda r: [r - 1, r - 90, r - 4500]),
    "ragged": (6200, lambda r: [r - 1, r - 61] + [r - 2100] * (r % 3 == 0) + [0] * (r % 31 == 0)),
    "xt3d": (3000, lambda r: [r - o for o in (1, 2, 49, 50, 51, 99, 100, 101, 1000, 1050, 1051)]),
}


@pytest.mark.parametrize("rows", [1, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("name", PATTERNS)
def test_plan_bitexact(plans, name, rows):
    n, lower = PATTERNS[name]
    iapc, japc, apc = factor_pattern(n, lower, seed=n)
    v = np.random.default_rng(rows).standard_normal(n)
    z, _ = walk(plans, iapc, japc, apc, v, rows)
    np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, v, fma=True))


@pytest.mark.parametrize("w", [63, 64, 65, 127, 128, 254, 255, 256])
def test_wide_rows_bitexact(plans, w):
    """A full band: each row a level, so a slice, of its own."""
    n = 600
    iapc, japc, apc = factor_pattern(n, band(w), seed=w)
    v = np.random.default_rng(w).standard_normal(n)
    for rows in (512, 2048):
        z, info = walk(plans, iapc, japc, apc, v, rows)
        np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, v, fma=True))
        z32, _ = walk(plans, iapc, japc, apc, v, rows, fp32=True)
        # each row sums w products of at most max|z| / w: a few FP32 roundings
        # of the result's scale a row, which the 1/w factors damp
        assert np.max(np.abs(z32 - z)) <= 1e-4 * np.max(np.abs(z))


def test_cut_slices_and_halved_ranges(plans):
    """Levels of 32 rows and 128 entries, whose ring of full slices does not
    fit, in narrower slices; halos that only fit smaller ranges; and a plan
    that fits as it is, which stays with full slices."""
    v = np.random.default_rng(3).standard_normal(8192)
    iapc, japc, apc = factor_pattern(8192, lambda r: range(r - 32 * 128, r, 32), seed=1)
    z, info = walk(plans, iapc, japc, apc, v, 2048)
    np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, v, fma=True))
    for i in info:
        assert i["maxblock"] <= 16 * 1024 and i["slices"] > 8192 // 32
    n = 40000
    u = np.random.default_rng(4).standard_normal(n)
    iapc, japc, apc = factor_pattern(n, lambda r: [r - 1, r - 8200, r - 16400, r - 24600], seed=2)
    z, info = walk(plans, iapc, japc, apc, u, 8192)
    np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, u, fma=True))
    assert all(i["R"] == 4096 for i in info)
    iapc, japc, apc = factor_pattern(3200, lambda r: range(r - 32 * 60, r, 32), seed=1)
    z, info = walk(plans, iapc, japc, apc, v[:3200], 2048)
    np.testing.assert_array_equal(z, oracle.ilu0a(apc, iapc, japc, v[:3200], fma=True))
    assert all(i["slices"] == 100 for i in info)


@pytest.mark.parametrize("forward", [1, 0])
def test_no_memory_is_no_plan(plans, forward):
    """Where an allocation of the plan fails, there is none, and the caller sweeps
    without: no exception leaves the library."""
    n, lower = PATTERNS["grid"]
    iapc, japc, apc = factor_pattern(n, lower, seed=n)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    results = {plans.range_starved(n, p(iapc), p(japc), japc.size, forward, 2048, C.c_longlong(1 << k))
               for k in range(2, 28)}
    assert results == {0, 1}
