"""What the library allocates, copies and launches, and where, on a stand-in for
the CUDA runtime that writes it down (c_abi/host_cudart.cpp): no GPU."""
import ctypes as C
import re
import shutil
import subprocess
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import pytest

from modflow6_gb300 import _lib
from modflow6_gb300.ensemble import EnsembleLinear
from modflow6_gb300.ims import GENERAL, ImsLinear, ImsLinearSettings
from test_gpu_batch_products import grid

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def hostlib(tmp_path_factory):
    """The library's own objects, linked with the stand-in."""
    if shutil.which("nvcc") is None or shutil.which("g++") is None:
        pytest.skip("nvcc or g++ not available")
    from modflow6_gb300 import build
    build.build()
    out = tmp_path_factory.mktemp("host") / "libhost.so"
    cuda = Path(shutil.which("nvcc")).resolve().parents[1]
    objs = [str(build.OBJ / (s.stem + ".o")) for s in build.sources()]
    cmd = ["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", str(cuda / "include"), "-o", str(out),
           str(ROOT / "tests" / "c_abi" / "host_cudart.cpp"), *objs, "-Wl,-Bsymbolic", "-Wl,-z,defs"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    lib = C.CDLL(str(out))
    for name, (res, args) in _lib._SIGS.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    lib.host_trace.restype = C.c_char_p
    lib.host_bytes.restype = C.c_longlong
    return lib


@pytest.fixture
def host(hostlib, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", hostlib)
    hostlib.host_set_device(0)
    hostlib.host_trace_clear()
    yield hostlib
    hostlib.host_set_device(0)


def trace(host):
    """The calls so far, kernels by their plain names; and a fresh trace."""
    lines = host.host_trace().decode().splitlines()
    host.host_trace_clear()
    return [re.sub(r"_ZN\S*?(\d+)(k_[a-z0-9_]+)\S*", lambda m: m.group(2)[:int(m.group(1))], l) for l in lines]


def launches(lines):
    return [l.split()[2] for l in lines if l.startswith("launch ")]


def band_pattern(n, offsets):
    """A symmetric matrix of the given band offsets, diagonal first."""
    ia, ja, a = np.zeros(n + 1, np.int32), [], []
    for r in range(n):
        row = sorted(c for o in offsets for c in (r - o, r + o) if 0 <= c < n)
        ja += [r] + row
        a += [-(len(row) + 1.0)] + [1.0] * len(row)
        ia[r + 1] = len(ja)
    return ia, np.array(ja, np.int32), np.array(a)


def optins(lines, device):
    return {l.split()[2]: int(l.split()[3]) for l in lines if l.startswith(f"optin {device} ")}


def test_shared_memory_is_asked_for_on_each_device(host):
    """A kernel's dynamic shared memory above 48 KB is a setting of the device
    it runs on: handles on two devices of a process each ask for theirs."""
    n = 6000
    ia, ja, a = band_pattern(n, list(range(100, 109)) + list(range(2000, 2009)))
    di, dj, da = band_pattern(n, [1, 50])
    asked = {}
    for device in (0, 1, 0):
        host.host_set_device(device)
        net = C.c_void_p()
        assert host.gbmpnn_create(n, dj.size, _lib.iptr(di), _lib.iptr(dj), 1, C.byref(net)) == 0
        x = np.zeros(n * 16, np.float32).ctypes.data_as(C.c_void_p)
        y = np.zeros(n, np.float32).ctypes.data_as(C.c_void_p)
        assert host.gbmpnn_forward(net, x, y) == 0
        assert host.gbmpnn_gradients(net, x, y, y, 1.0, None, None) == 0
        host.gbmpnn_destroy(net)
        z = np.zeros(n)
        ims = ImsLinear(ImsLinearSettings(structure=GENERAL)).imslinear_allocate(n, ia, ja)
        assert host.gbims_factor(ims._h, _lib.dptr(a), None) == 0
        assert host.gbims_precondition(ims._h, _lib.dptr(z), _lib.dptr(z)) == 0
        gi, gj, ga = grid(2, 40, 75, np.random.default_rng(0))
        ims = ImsLinear(ImsLinearSettings(structure=(2, 40, 75))).imslinear_allocate(n, gi, gj)
        assert host.gbims_factor(ims._h, _lib.dptr(ga), None) == 0
        assert host.gbims_set_tuning(ims._h, 6, 0, -1) == 0  # the tiling of two blocks an SM
        assert host.gbims_precondition(ims._h, _lib.dptr(z), _lib.dptr(z)) == 0
        lines = trace(host)
        ran = {l.split()[2]: int(l.split()[4]) for l in lines if l.startswith("launch ")}
        big = {k: b for k, b in ran.items() if b > 48 * 1024}
        assert {"k_layer", "k_layer_bwd", "k_range_sweep", "k_dia7_sweep"} <= set(big)
        asked.setdefault(device, {}).update(optins(lines, device))
        assert all(asked[device].get(k, 0) >= b for k, b in big.items()), (device, big, asked)


@pytest.mark.parametrize("shapes", [None, [(1, 5, 6)] * 3], ids=["general", "grids"])
def test_batch_calls_clear_the_control_blocks(host, shapes):
    """The members' control blocks gate a batch's products and sweeps: they are
    cleared when the handle is made and before a call outside a solve."""
    members = [grid(1, 5, 6, np.random.default_rng(0))] * 3
    ia = np.concatenate([[0]] + [i[1:] + k * i[-1] for k, (i, _, _) in enumerate(members)]).astype(np.int32)
    ja = np.concatenate([j + 30 * k for k, (_, j, _) in enumerate(members)]).astype(np.int32)
    a = np.concatenate([m[2] for m in members])
    v, t = np.zeros(90), _lib.GbimsKernelTimes()
    ens = EnsembleLinear(ImsLinearSettings()).allocate(np.array([0, 30, 60, 90], np.int32), ia, ja, shapes)
    assert host.gbims_factor(ens._h, _lib.dptr(a), None) == 0
    trace(host)
    for call in (lambda: host.gbims_matvec(ens._h, _lib.dptr(v), _lib.dptr(v)),
                 lambda: host.gbims_precondition(ens._h, _lib.dptr(v), _lib.dptr(v)),
                 lambda: host.gbims_time_kernels(ens._h, 1, C.byref(t))):
        assert call() == 0
        lines = trace(host)
        first = next(i for i, l in enumerate(lines) if "spmv" in l or "sweep" in l)
        assert any(l.startswith("memset") for l in lines[:first]), lines
    ens.close()


@pytest.mark.parametrize("level", [0, 3], ids=["ilu0", "ilut"])
def test_plans_are_sent_on_the_handles_stream(host, level):
    """Work on the handle's stream, which does not wait for the legacy stream,
    reads the sweeps' plans and level schedules: their copies go on it too."""
    ia, ja, a = band_pattern(3000, [1, 50])
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, level=level)).imslinear_allocate(3000, ia, ja)
    trace(host)
    assert host.gbims_factor(ims._h, _lib.dptr(a), None) == 0
    assert host.gbims_set_tuning(ims._h, -1, 0, 0) == 0
    assert host.gbims_set_tuning(ims._h, -1, 0, 1) == 0
    assert host.gbims_factor(ims._h, _lib.dptr(a), None) == 0
    lines = trace(host)
    assert level or "k_range_fill" in launches(lines)
    assert not [l for l in lines if re.match(r"(memcpy|memset) 0 ", l)]


def test_creation_is_done_when_it_returns(host):
    """What the calls that make a handle clear and copy on the legacy stream is
    waited for before the handle's own stream, which does not wait for it, reads
    it: zeroed hand-over words above all."""
    gi, gj, ga = grid(2, 6, 7, np.random.default_rng(0))
    gi, gj = gi.astype(np.int32), gj.astype(np.int32)
    bi, bj, ba = band_pattern(84, [1, 7])
    v = np.zeros(84)

    def check(call):
        trace(host)
        call()
        pending = None
        for l in trace(host):
            if re.match(r"(memcpy|memset) 0 ", l):
                pending = l
            elif l == "synchronize 0":
                pending = None
            else:
                assert not (pending and l.startswith("launch ")), (pending, l)

    def linear(settings, ia, ja, a, *more):
        ims = ImsLinear(settings).imslinear_allocate(84, ia, ja)
        for call in more:
            assert call(ims._h) == 0
        assert host.gbims_factor(ims._h, _lib.dptr(a), None) == 0
        assert host.gbims_precondition(ims._h, _lib.dptr(v), _lib.dptr(v)) == 0

    check(lambda: linear(ImsLinearSettings(structure=GENERAL), bi, bj, ba))
    check(lambda: linear(ImsLinearSettings(level=3), bi, bj, ba))
    check(lambda: linear(ImsLinearSettings(structure=(2, 6, 7)), gi, gj, ga))
    start = np.array([0, 40, 84], np.int32)
    check(lambda: linear(ImsLinearSettings(structure=GENERAL), bi, bj, ba,
                         lambda h: host.gbims_set_inner_records(h, 5, 2, _lib.iptr(start))))

    def batch(shapes):
        ens = EnsembleLinear(ImsLinearSettings()).allocate(np.array([0, 84], np.int32), gi, gj, shapes)
        assert host.gbims_factor(ens._h, _lib.dptr(ga), None) == 0

    check(lambda: batch(None))
    check(lambda: batch([(2, 6, 7)]))

    def network():
        net = C.c_void_p()
        assert host.gbmpnn_create(84, bj.size, _lib.iptr(bi), _lib.iptr(bj), 1, C.byref(net)) == 0
        assert host.gbmpnn_set_params(net, f) == 0
        host.gbmpnn_destroy(net)

    f = np.zeros(200000, np.float32).ctypes.data_as(C.POINTER(C.c_float))
    check(network)


def solve_launches(host, ims, a):
    n = ims.neq
    trace(host)
    ims.imslinear_apply(a.copy(), np.ones(n), np.zeros(n))
    return trace(host)


def test_refused_and_failed_tuning_leave_no_stale_loop(host):
    """A solve's captured loop sweeps with what the factorisation has just
    filled, also after a tuning that was refused or that failed half way."""
    ia, ja, a = band_pattern(3000, [1, 50])
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1)).imslinear_allocate(3000, ia, ja)
    first = set(launches(solve_launches(host, ims, a)))
    assert {"k_range_fill", "k_range_sweep"} <= first
    # refused for its tiling: nothing of it is taken
    assert host.gbims_set_tuning(ims._h, 99, 0, 0) == _lib.GBIMS_ERR_ARG
    assert set(launches(solve_launches(host, ims, a))) == first
    # a tuning that fails after it has replaced the plans: captured again
    host.host_fail_copy(4)
    assert host.gbims_autotune(ims._h, 1, C.byref(_lib.GbimsTuning())) == _lib.GBIMS_ERR_CUDA
    lines = solve_launches(host, ims, a)
    again = set(launches(lines))
    assert "capture" in lines and ("k_range_fill" in again) == ("k_range_sweep" in again) != ("k_ilu_sweep_sf" in again)
    assert host.gbims_set_tuning(ims._h, -1, 0, 0) == 0
    lines = launches(solve_launches(host, ims, a))
    assert "k_ilu_fwd_level" in lines and not {"k_range_fill", "k_range_sweep"} & set(lines)


def test_memory_of_a_batch_of_grids(host):
    """A batch of one grid holds what a handle of the grid does, besides its
    chunks' and members' few words: no words by nonzero, no level schedule."""
    ia, ja, a = grid(4, 64, 96, np.random.default_rng(0))
    n = ia.size - 1
    before = host.host_bytes()
    one = ImsLinear(ImsLinearSettings(structure=(4, 64, 96))).imslinear_allocate(n, ia, ja)
    single = host.host_bytes() - before
    before = host.host_bytes()
    ens = EnsembleLinear(ImsLinearSettings()).allocate(np.array([0, n], np.int32), ia.astype(np.int32),
                                                       ja.astype(np.int32), [(4, 64, 96)])
    batch = host.host_bytes() - before
    assert abs(batch - single) <= 16 * 1024
    ens.close()
    one.imslinear_da()
    assert host.host_bytes() == before - single


@pytest.mark.parametrize("accel", [1, 2])
@pytest.mark.parametrize("precision", [_lib.GBIMS_FP64, _lib.GBIMS_MIXED], ids=["fp64", "mixed"])
def test_tuned_loop_keeps_its_form(host, precision, accel):
    """The tuner leaves the reduction grid of a system with fused products alone,
    and a smaller grid that is set leaves the loop's kernels as they are."""
    n = 60000
    ia, ja, a = band_pattern(n, [1, 300])
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1, ilinmeth=accel, precision=precision)
                    ).imslinear_allocate(n, ia, ja)
    first = launches(solve_launches(host, ims, a))
    assert "k_sell_spmv_fin" in first
    t = _lib.GbimsTuning()
    assert host.gbims_autotune(ims._h, 1, C.byref(t)) == 0
    assert t.reduction_blocks == (n + 255) // 256  # fewer blocks are faster on the stand-in
    assert host.gbims_set_tuning(ims._h, -1, 0, 1) == 0
    assert launches(solve_launches(host, ims, a)) == first
    assert host.gbims_set_tuning(ims._h, -1, 17, -1) == 0
    assert launches(solve_launches(host, ims, a)) == first


@pytest.mark.parametrize("accel", [1, 2])
def test_fused_products_by_size(host, accel):
    """Fused on full grids up to 311,296 rows, and on general patterns up to two
    million entries (BiCGSTAB three)."""
    def products(n, ia, ja, a, structure):
        ims = ImsLinear(ImsLinearSettings(structure=structure, iter1=1, ilinmeth=accel)).imslinear_allocate(n, ia, ja)
        return {k for k in launches(solve_launches(host, ims, a)) if "spmv" in k}
    most = 1000000 * (1 + accel)
    below, above = most // 63, most // 63 + 100  # rows of 63 entries, fewer at both ends
    for n, offsets, fused in ((32000, [1, 40], True), (below, range(1, 32), True), (above, range(1, 32), False)):
        ia, ja, a = band_pattern(n, offsets)
        assert (ja.size <= most) == fused
        assert ("k_sell_spmv_fin" in products(n, ia, ja, a, GENERAL)) == fused
    for shape, fused in (((1, 608, 512), True), ((1, 608, 513), False)):
        ia, ja, a = grid(*shape, np.random.default_rng(0))
        ia, ja = ia.astype(np.int32), ja.astype(np.int32)
        assert ("k_dia7_spmv_fin" in products(ia.size - 1, ia, ja, a, shape)) == fused


def shuffled_grid(nrow, ncol, seed):
    """A one-layer grid whose cells are numbered in random order."""
    ia, ja, a = grid(1, nrow, ncol, np.random.default_rng(seed))
    n = ia.size - 1
    new = np.random.default_rng(seed + 1).permutation(n)
    old = np.argsort(new)
    pa, pj, pv = np.zeros(n + 1, np.int32), [], []
    for r in range(n):
        k = np.arange(ia[old[r]], ia[old[r] + 1])
        c = new[ja[k]]
        o = np.argsort(np.where(c == r, -1, c))
        pj += list(c[o])
        pv += list(a[k[o]])
        pa[r + 1] = len(pj)
    return pa, np.array(pj, np.int32), np.array(pv)


def test_sweeps_by_pattern(host):
    """Over ranges where rows depend on near rows, sync-free where levels are few
    and dependencies far; ILUT's by each factor's pattern (none here: kernels do
    not run); what the tuner finds best stays."""
    ia, ja, a = shuffled_grid(60, 70, 1)
    n = ia.size - 1
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1)).imslinear_allocate(n, ia, ja)
    L = set(launches(solve_launches(host, ims, a)))
    assert "k_ilu_sweep_sf" in L and not {"k_range_sweep", "k_range_fill"} & L
    assert host.gbims_set_tuning(ims._h, -1, 0, 0) == 0
    assert "k_ilu_fwd_level" in launches(solve_launches(host, ims, a))
    assert host.gbims_set_tuning(ims._h, -1, 0, 1) == 0
    assert "k_ilu_sweep_sf" in launches(solve_launches(host, ims, a))
    t = _lib.GbimsTuning()
    assert host.gbims_autotune(ims._h, 1, C.byref(t)) == 0
    assert t.level_mode == 1 and t.ncandidates == 6
    assert "k_range_sweep" in launches(solve_launches(host, ims, a))  # fewer blocks are faster on the stand-in
    ia, ja, a = band_pattern(3000, [1, 50])
    ims = ImsLinear(ImsLinearSettings(structure=GENERAL, iter1=1)).imslinear_allocate(3000, ia, ja)
    assert "k_range_sweep" in launches(solve_launches(host, ims, a))
    ims = ImsLinear(ImsLinearSettings(level=3, iter1=1)).imslinear_allocate(3000, ia, ja)
    assert "k_ilu_sweep_sf" in launches(solve_launches(host, ims, a))
