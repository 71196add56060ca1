"""Performance cases of the framework: what a user of it has it do, through
its public entry points.

Each case is one pass of one of these calls:

* "gwf": `GwfSolution` (restart, one time step to closure, the heads): the
  device-resident solution of a DIS, DISV or DISU model (PCG + ILU0), of a
  model with the full conductivity tensor (XT3D, BiCGSTAB + ILU0), or of a
  convertible transient Newton model (BiCGSTAB + ILU0, delta-bar-delta
  under-relaxation);
* "linear": `ImsLinear.imslinear_apply` on a linear system in host arrays,
  as MODFLOW 6 hands it to its linear solver each outer iteration (`host`),
  or `ImsLinear.apply_device` on one in device memory;
* "ensemble": `EnsembleLinear.apply_device`, many uneven DIS systems at once;
* "network": the warm-start network on the graph of a DIS matrix:
  `WarmStartNet.predict`, or `WarmStartNet.gradients` of the squared error.

The models are synthetic (lognormal K, constant heads on two faces, wells)
in the sizes of the repository's workloads and tests or between them.  The
closures are tight, so that the heads that come back are the solution of the
system and not the point at which an iteration happened to stop.
"""
import math

import numpy as np
import torch

DEV = "cuda"


def listed():
    return [
        # a small demonstration or test model (the size of the package tests'
        # grids): launches and latency are all there is
        dict(name="gwf_dis_1x20x30", kind="gwf", grid="dis", nlay=1, nrow=20, ncol=30, precision="fp64"),
        # the 100 x 100 single-layer areal model, the commonest small size
        dict(name="gwf_dis_1x100x100", kind="gwf", grid="dis", nlay=1, nrow=100, ncol=100, precision="fp64"),
        # a large regional model: 3.6 million cells in ten layers
        dict(name="gwf_dis_10x600x600", kind="gwf", grid="dis", nlay=10, nrow=600, ncol=600, precision="fp64"),
        # a mid-sized model in the mixed-precision form
        dict(name="gwf_dis_mixed_5x255x310", kind="gwf", grid="dis", nlay=5, nrow=255, ncol=310,
             precision="mixed"),
        # one step of a transient water-table (NEWTON) model
        dict(name="gwf_newton_5x90x90", kind="gwf", grid="newton", nlay=5, nrow=90, ncol=90,
             precision="fp64"),
        # an unstructured (DISV hexagon) model of 90,000 cells
        dict(name="gwf_disv_4x150x150", kind="gwf", grid="disv", nlay=4, nrow=150, ncol=150,
             precision="fp64"),
        # a model with the full conductivity tensor: the wide matrix rows
        dict(name="gwf_xt3d_3x70x70", kind="gwf", grid="xt3d", nlay=3, nrow=70, ncol=70, precision="fp64"),
        # the drop-in linear solver called with MODFLOW 6's host arrays
        dict(name="linear_host_10x200x200", kind="linear", nlay=10, nrow=200, ncol=200, host=True,
             complexity="SIMPLE"),
        # the COMPLEX preset (BiCGSTAB + ILUT) on a system in device memory
        dict(name="linear_ilut_6x60x60", kind="linear", nlay=6, nrow=60, ncol=60, host=False,
             complexity="COMPLEX"),
        # an ensemble of uneven models, every member to its own closure
        dict(name="ensemble_24", kind="ensemble", members=24, low=50, high=250, shuffle=0),
        # the warm-start network on the transient 256 x 256 x 3 workload:
        # one guess, and one training gradient
        dict(name="network_predict_3x256x256", kind="network", nlay=3, nrow=256, ncol=256, train=False),
        dict(name="network_train_3x256x256", kind="network", nlay=3, nrow=256, ncol=256, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a grid of any of the kinds, its sizes spread over the
    logarithm of their range, odd ones among them."""
    kind = rng.choice(["dis", "dis", "disv", "disu", "newton", "xt3d", "linear", "ilut", "ensemble",
                       "network"])
    if kind == "dis":
        r, c = _log(rng, 16, 500), _log(rng, 16, 500)
        return dict(kind="gwf", grid="dis", nlay=rng.randint(1, 10), nrow=r, ncol=c,
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "disv":
        return dict(kind="gwf", grid="disv", nlay=rng.randint(1, 5), nrow=_log(rng, 12, 160),
                    ncol=_log(rng, 12, 160), precision="fp64")
    if kind == "disu":
        return dict(kind="gwf", grid="disu", nlay=rng.randint(1, 4), nrow=_log(rng, 12, 90),
                    ncol=_log(rng, 12, 90), precision="fp64")
    if kind == "newton":
        return dict(kind="gwf", grid="newton", nlay=rng.randint(1, 5), nrow=_log(rng, 16, 100),
                    ncol=_log(rng, 16, 100), precision="fp64")
    if kind == "xt3d":
        return dict(kind="gwf", grid="xt3d", nlay=rng.randint(1, 4), nrow=_log(rng, 12, 70),
                    ncol=_log(rng, 12, 70), precision="fp64")
    if kind == "linear":
        return dict(kind="linear", nlay=rng.randint(1, 10), nrow=_log(rng, 20, 220),
                    ncol=_log(rng, 20, 220), host=rng.random() < 0.5,
                    complexity=rng.choice(["SIMPLE", "MODERATE"]))
    if kind == "ilut":
        return dict(kind="linear", nlay=rng.randint(1, 6), nrow=_log(rng, 12, 60),
                    ncol=_log(rng, 12, 60), host=rng.random() < 0.5, complexity="COMPLEX")
    if kind == "ensemble":
        return dict(kind="ensemble", members=_log(rng, 2, 32), low=_log(rng, 12, 50),
                    high=_log(rng, 60, 200), shuffle=rng.randint(1, 1 << 20))
    return dict(kind="network", nlay=rng.randint(1, 4), nrow=_log(rng, 24, 300), ncol=_log(rng, 24, 300),
                train=rng.random() < 0.5)


# -- inputs ------------------------------------------------------------------


def _field(rng, nlay, nrow, ncol, sigma, corr):
    """Lognormal K per layer: Gaussian-filtered white noise (correlation
    length `corr` cells, in the Fourier domain), standardised."""
    fy = np.fft.fftfreq(nrow)[:, None]
    fx = np.fft.rfftfreq(ncol)[None, :]
    h = np.exp(-2.0 * (np.pi * corr) ** 2 * (fy * fy + fx * fx))
    out = []
    for _ in range(nlay):
        w = np.fft.irfft2(np.fft.rfft2(rng.standard_normal((nrow, ncol))) * h, s=(nrow, ncol))
        sd = w.std()
        w = (w - w.mean()) / (sd if sd > 0 else 1.0)
        out.append(np.exp(sigma * w).ravel())
    return np.concatenate(out)


def _faces(nlay, nrow, ncol):
    k, i = np.meshgrid(np.arange(nlay), np.arange(nrow), indexing="ij")
    west = (k * nrow * ncol + i * ncol).ravel()
    return west.astype(np.int32), (west + ncol - 1).astype(np.int32)


def _dis_model(nlay, nrow, ncol, seed, sigma=1.0, corr=8.0, hwest=20.0, heast=0.0, wells=True):
    """Confined steady DIS model: 10 m cells and layers, CHD on the west and
    east faces, wells in one cell of 2,000."""
    from modflow6_gb300.dis import GwfDisModel
    rng = np.random.default_rng([seed, nlay, nrow, ncol])
    nrc, n = nrow * ncol, nlay * nrow * ncol
    k = _field(rng, nlay, nrow, ncol, sigma, corr)
    botm = np.repeat(10.0 * nlay - 10.0 * np.arange(1, nlay + 1), nrc)
    m = GwfDisModel(nlay, nrow, ncol, np.full(ncol, 10.0), np.full(nrow, 10.0),
                    np.full(nrc, 10.0 * nlay), botm, k, 0.1 * k, np.zeros(n, np.int32),
                    np.full(n, 0.5 * (hwest + heast)))
    west, east = _faces(nlay, nrow, ncol)
    m.chd_node = np.concatenate([west, east])
    m.chd_head = np.concatenate([np.full(west.size, hwest), np.full(east.size, heast)])
    if wells:
        cand = np.ones(n, bool)
        cand[m.chd_node] = False
        cand = np.flatnonzero(cand)
        m.wel_node = np.sort(rng.choice(cand, size=max(1, n // 2000), replace=False)).astype(np.int32)
        m.wel_q = rng.uniform(-50.0, -5.0, m.wel_node.size)
    return m


def _newton_model(nlay, nrow, ncol, seed):
    """Convertible transient model: 10 m cells, sloping bottom, recharge,
    wells, specific yield 0.15."""
    m = _dis_model(nlay, nrow, ncol, seed, wells=False)
    rng = np.random.default_rng([seed, 7])
    n, nrc = m.nodes, nrow * ncol
    bottom = np.tile(np.linspace(0.0, -40.0, ncol), nrow)
    m.top = np.full(nrc, 50.0)
    m.botm = np.concatenate([50.0 + (f + 1) / nlay * (bottom - 50.0) for f in range(nlay)])
    m.k33 = m.k11.copy()
    m.icelltype = np.ones(n, np.int32)
    m.strt = np.full(n, 45.0)
    m.ss, m.sy = np.full(n, 1.0e-5), np.full(n, 0.15)
    m.chd_node, m.chd_head = np.zeros(0, np.int32), np.zeros(0)
    m.inewton = 1
    m.wel_node = np.sort(rng.choice(n, size=max(1, n // 600), replace=False)).astype(np.int32)
    m.wel_q = rng.uniform(-200.0, 0.0, m.wel_node.size)
    m.rch_node = np.arange(nrc, dtype=np.int32)
    m.rch_rate = rng.uniform(0.0, 5.0e-4, nrc)
    return m


def _model(case, seed):
    nlay, nrow, ncol, grid = case["nlay"], case["nrow"], case["ncol"], case["grid"]
    if grid == "dis":
        return _dis_model(nlay, nrow, ncol, seed)
    if grid == "newton":
        return _newton_model(nlay, nrow, ncol, seed)
    if grid == "disv":
        from modflow6_gb300.disv import make_disv_model
        return make_disv_model(nlay, ncol, nrow, seed=seed % (1 << 31))
    if grid == "disu":
        from modflow6_gb300.disu import make_disu_model
        return make_disu_model(nlay, nrow, ncol, seed=seed % (1 << 31))
    m = _dis_model(nlay, nrow, ncol, seed, hwest=28.0, heast=22.0)
    n = m.nodes
    m.ixt3d, m.k22, m.k33 = 1, 0.2 * m.k11, 0.05 * m.k11
    m.angle1, m.angle2, m.angle3 = np.full(n, 30.0), np.full(n, 15.0), np.full(n, 5.0)
    return m


def _system(m):
    """The linear system of a confined steady DIS model as the solver is
    handed it (constant heads eliminated): (ia, ja, amat, rhs, x0), in
    numpy, with the two-point harmonic conductances of the grid's faces."""
    nlay, nrow, ncol = m.nlay, m.nrow, m.ncol
    n = m.nodes
    k11 = m.k11.reshape(nlay, nrow, ncol)
    k33 = m.k33.reshape(nlay, nrow, ncol)
    z = 10.0
    harm = lambda a, b: 2.0 * a * b / (a + b)
    cr = np.zeros((nlay, nrow, ncol))  # to the next column
    cf = np.zeros((nlay, nrow, ncol))  # to the next row
    cv = np.zeros((nlay, nrow, ncol))  # to the next layer
    cr[:, :, :-1] = z * harm(k11[:, :, :-1], k11[:, :, 1:])
    cf[:, :-1, :] = z * harm(k11[:, :-1, :], k11[:, 1:, :])
    cv[:-1] = 10.0 * harm(k33[:-1], k33[1:])
    chd = np.zeros(n, bool)
    chd[m.chd_node] = True
    head = np.zeros(n)
    head[m.chd_node] = m.chd_head
    node = np.arange(n).reshape(nlay, nrow, ncol)
    up = np.zeros_like(cv); up[1:] = cv[:-1]
    back = np.zeros_like(cf); back[:, 1:, :] = cf[:, :-1, :]
    left = np.zeros_like(cr); left[:, :, 1:] = cr[:, :, :-1]
    offs = (-nrow * ncol, -ncol, -1, 1, ncol, nrow * ncol)
    kk, ii, jj = np.indices((nlay, nrow, ncol))
    has = (kk > 0, ii > 0, jj > 0, jj < ncol - 1, ii < nrow - 1, kk < nlay - 1)
    has = np.stack([h.ravel() for h in has])
    cond = np.stack([c.ravel() for c in (up, back, left, cr, cf, cv)])
    ia = np.zeros(n + 1, np.int64)
    np.cumsum(1 + has.sum(axis=0), out=ia[1:])
    ja = np.empty(ia[-1], np.int32)
    amat = np.empty(ia[-1])
    rhs = np.zeros(n)
    np.add.at(rhs, m.wel_node, -m.wel_q)
    ja[ia[:-1]] = node.ravel()
    amat[ia[:-1]] = np.where(chd, 1.0, -cond.sum(axis=0))
    rhs[chd] = head[chd]
    pos = ia[:-1] + 1
    for d in range(6):
        r = np.flatnonzero(has[d])
        c = r + offs[d]
        ja[pos[r]] = c
        # a row or column of a constant head leaves the matrix; its product
        # with the head moves to the right-hand side
        amat[pos[r]] = np.where(chd[r] | chd[c], 0.0, cond[d][r])
        e = ~chd[r] & chd[c]
        rhs[r[e]] -= cond[d][r[e]] * head[c[e]]
        pos = pos + has[d]
    x0 = m.strt.copy()
    x0[chd] = head[chd]
    return ia.astype(np.int32), ja, amat, rhs, x0


def _ensemble_models(case, seed):
    rng = np.random.default_rng([case["members"], case["low"], case["high"], case["shuffle"]])
    out = []
    for i in range(case["members"]):
        nrow, ncol = (int(v) for v in rng.integers(case["low"], case["high"] + 1, size=2))
        nlay = int(rng.integers(1, 6))
        out.append(_dis_model(nlay, nrow, ncol, seed * 1000 + i, sigma=float(rng.uniform(0.5, 1.5)),
                              hwest=float(rng.uniform(10.0, 20.0)), heast=float(rng.uniform(0.0, 10.0)),
                              wells=False))
    return out


def _concat(systems):
    row = np.cumsum([0] + [s[4].size for s in systems])
    nz = np.cumsum([0] + [s[1].size for s in systems])
    ia = np.concatenate([s[0][:-1] + nz[i] for i, s in enumerate(systems)] + [[nz[-1]]]).astype(np.int32)
    ja = np.concatenate([s[1] + row[i] for i, s in enumerate(systems)]).astype(np.int32)
    amat, rhs, x0 = (np.concatenate([s[q] for s in systems]) for q in (2, 3, 4))
    return row.astype(np.int32), ia, ja, amat, rhs, x0


def _network_inputs(case, seed):
    """Graph matrix (a DIS system), network parameters at the size of a
    trained network's, features in their standardised units, targets."""
    m = _dis_model(case["nlay"], case["nrow"], case["ncol"], seed, hwest=25.0)
    ia, ja, amat, _, _ = _system(m)
    rng = np.random.default_rng([seed, 11])
    n = m.nodes
    parts = [rng.standard_normal(16 * 64) * 0.35, np.zeros(64)]
    for _ in range(8):
        parts += [rng.standard_normal(128 * 64) * 0.06, rng.standard_normal(64) * 0.01]
    parts += [rng.standard_normal(64) * 0.12, np.zeros(1)]
    p = np.concatenate(parts).astype(np.float32)
    x = np.zeros((n, 16), np.float32)
    x[:, 0] = np.log(m.k11)
    x[:, 1] = rng.standard_normal(n)
    x[m.wel_node, 2] = m.wel_q / 100.0
    x[m.chd_node, 3] = 1.0
    x[:, 4] = np.repeat(np.arange(m.nlay) / max(1, m.nlay - 1), m.nrow * m.ncol)
    x[:, 5] = 1.0
    x[:, 6] = rng.standard_normal(n) * 0.5
    mask = np.ones(n, np.float32)
    mask[m.chd_node] = 0.0
    t = rng.standard_normal(n).astype(np.float32) * mask
    return m, ia, ja, amat, p, x, t, mask


# -- settings ----------------------------------------------------------------

_PCG = dict(dvclose=1e-9, rclose=2e-9)
_GENERAL = dict(dvclose=1e-9, rclose=1e-8)
_LINEAR = dict(
    SIMPLE=dict(iter1=5000, **_PCG),
    MODERATE=dict(iter1=5000, **_PCG),
    COMPLEX=dict(iter1=2000, **_PCG),
)


def _delt(case):
    return 2.0 if case["grid"] == "newton" else 1.0


def prepare(case, seed):
    from modflow6_gb300 import _lib
    from modflow6_gb300.ims import ImsLinear, ImsLinearSettings
    if case["kind"] == "gwf":
        from modflow6_gb300.solution import GwfSolution, Nonlinear
        m = _model(case, seed)
        grid = case["grid"]
        kw = dict(_PCG if grid == "dis" else _GENERAL, iter1=20000, ilinmeth=2 if grid in ("newton", "xt3d") else 1,
                  precision=_lib.GBIMS_MIXED if case["precision"] == "mixed" else _lib.GBIMS_FP64)
        if case["precision"] == "mixed":
            kw.update(rclose=1e-9)
        nl = Nonlinear(dvclose=1e-8, mxiter=25)
        if grid == "newton":
            # the MODERATE preset's under-relaxation
            nl = Nonlinear.preset("MODERATE", dvclose=1e-5, mxiter=100)
        return dict(sol=GwfSolution(m, ImsLinearSettings(**kw), nl), delt=_delt(case))
    if case["kind"] == "linear":
        m = _dis_model(case["nlay"], case["nrow"], case["ncol"], seed)
        ia, ja, amat, rhs, x0 = _system(m)
        s = ImsLinearSettings.preset_config(case["complexity"], **_LINEAR[case["complexity"]])
        st = dict(ims=ImsLinear(s).imslinear_allocate(m.nodes, ia, ja))
        if case["host"]:
            st.update(amat=amat, rhs=rhs, x0=x0)
        else:
            st.update({k: torch.from_numpy(v).to(DEV) for k, v in
                       (("amat", amat), ("rhs", rhs), ("x0", x0))})
            st["x"] = torch.empty_like(st["x0"])
            torch.cuda.synchronize()
        return st
    if case["kind"] == "ensemble":
        from modflow6_gb300.ensemble import EnsembleLinear
        models = _ensemble_models(case, seed)
        row, ia, ja, amat, rhs, x0 = _concat([_system(m) for m in models])
        ens = EnsembleLinear(ImsLinearSettings(iter1=20000, ilinmeth=1, **_PCG)).allocate(
            row, ia, ja, [(m.nlay, m.nrow, m.ncol) for m in models])
        st = {k: torch.from_numpy(v).to(DEV) for k, v in (("amat", amat), ("rhs", rhs), ("x0", x0))}
        st.update(ens=ens, x=torch.empty_like(st["x0"]))
        torch.cuda.synchronize()
        return st
    from modflow6_gb300.warmstart import Graph, WarmStartNet
    m, ia, ja, amat, p, x, t, mask = _network_inputs(case, seed)
    net = WarmStartNet(Graph(m), seed=0)
    net.params = p
    d_amat = torch.from_numpy(amat).to(DEV)
    st = dict(net=net, amat=d_amat, x=torch.from_numpy(x).to(DEV), t=torch.from_numpy(t).to(DEV),
              mask=torch.from_numpy(mask).to(DEV), inv=1.0 / float(mask.sum()), train=case["train"])
    torch.cuda.synchronize()
    net.set_graph(d_amat)
    return st


def run(state):
    if "sol" in state:
        sol = state["sol"]
        sol.restart()
        sol.timestep(1, 1, state["delt"])
        return sol.heads
    if "ims" in state:
        if isinstance(state["x0"], np.ndarray):
            x = state["x0"].copy()
            state["ims"].imslinear_apply(state["amat"], state["rhs"], x)
            return x
        state["x"].copy_(state["x0"])
        torch.cuda.current_stream().synchronize()
        state["ims"].apply_device(state["amat"].data_ptr(), state["rhs"].data_ptr(),
                                  state["x"].data_ptr())
        return state["x"]
    if "ens" in state:
        state["x"].copy_(state["x0"])
        torch.cuda.current_stream().synchronize()
        state["ens"].apply_device(state["amat"].data_ptr(), state["rhs"].data_ptr(),
                                  state["x"].data_ptr())
        return state["x"]
    if state["train"]:
        loss, g = state["net"].gradients(state["x"], state["t"], state["mask"], state["inv"])
        return dict(loss=np.float32(loss), gradient=g)
    return state["net"].predict(state["x"])


# -- work --------------------------------------------------------------------


def _iterations(case):
    """Inner iterations that ILU0-preconditioned Krylov takes to the closures
    here, from the lengths of the grid."""
    long = max(case["nrow"], case["ncol"])
    if case["kind"] == "linear" and case["complexity"] != "SIMPLE":
        return 0.5 * long + 10
    if case.get("grid") == "newton":
        return 150
    return 2.0 * long + 20


def work(case):
    """One pass: per inner iteration the matrix, the factor and five vectors
    once each (the vectors a Krylov iteration has to read or write), and the
    products and sums of those entries; for the network, each layer's state
    read and written once and its matrix products."""
    if case["kind"] == "ensemble":
        rng = np.random.default_rng([case["members"], case["low"], case["high"], case["shuffle"]])
        b = f = 0.0
        for _ in range(case["members"]):
            nrow, ncol = (int(v) for v in rng.integers(case["low"], case["high"] + 1, size=2))
            nlay = int(rng.integers(1, 6))
            rng.uniform(), rng.uniform(), rng.uniform()
            it = 2.0 * max(nrow, ncol) + 20
            b += it * nlay * nrow * ncol * (14 + 5) * 8
            f += it * nlay * nrow * ncol * 40
        return dict(bytes=b, flops=f)
    n = case["nlay"] * case["nrow"] * case["ncol"]
    if case["kind"] == "network":
        flops = n * 2.0 * (16 * 64 + 8 * (128 * 64 + 7 * 64) + 64)
        byts = n * (16 + 1) * 4.0 + n * 7 * 4.0 * 8 + n * 64 * 4.0 * 2 * 8
        return dict(bytes=byts * (3 if case["train"] else 1), flops=flops * (3 if case["train"] else 1))
    width = {"xt3d": 23, "disv": 9}.get(case.get("grid"), 7)
    per = (2 * width + 5) * 8 * (0.5 if case.get("precision") == "mixed" else 1.0)
    it = _iterations(case)
    return dict(bytes=it * n * per, flops=it * n * (4.0 * width + 12))


# -- exact values ------------------------------------------------------------


def _solve64(ia, ja, amat, rhs, x0):
    """The solution of a system with constant heads eliminated, in 64 bits:
    conjugate gradients with a diagonal preconditioner, restarted from the
    true residual until it no longer falls."""
    n = rhs.size
    a = torch.sparse_csr_tensor(torch.from_numpy(ia.astype(np.int64)), torch.from_numpy(ja.astype(np.int64)),
                                torch.from_numpy(amat), size=(n, n)).to(DEV)
    diag = torch.from_numpy(amat[ia[:-1]]).to(DEV)
    b = torch.from_numpy(rhs).to(DEV)
    x = torch.from_numpy(x0).to(DEV).clone()
    # constant-head rows are 1 on a negative definite matrix: they are solved
    # already, so that their residual is zero and stays so
    best = float("inf")
    for _ in range(6):
        r = b - a @ x
        nr = float(r.norm())
        if nr == 0.0 or nr >= 0.5 * best:
            break
        best = nr
        z = r / diag
        p, rz = z.clone(), r @ z
        for it in range(1, 40001):
            q = a @ p
            al = rz / (p @ q)
            x += al * p
            r -= al * q
            z = r / diag
            new = r @ z
            p = z + (new / rz) * p
            rz = new
            if it % 100 == 0 and float(r.norm()) < 1e-6 * nr:
                break
    return x


def _grid_system(m):
    """The system of a confined steady DISV or DISU model from its
    connection list: conductance = width (or area) over the two half
    lengths' resistances."""
    con = m.connections()
    ia, ja, jas, ihc = (np.asarray(con[k], np.int64) for k in ("ia", "ja", "jas", "ihc"))
    n = ia.size - 1
    row = np.repeat(np.arange(n), np.diff(ia))
    off = ja != row
    s, r, c = jas[off], row[off], ja[off]
    low = r < c
    thick = m.cell_top - m.cell_bot
    l1 = np.where(low, con["cl1"][s], con["cl2"][s])
    l2 = np.where(low, con["cl2"][s], con["cl1"][s])
    w = con["hwva"][s]
    vert = ihc[s] == 0
    t1 = np.where(vert, m.k33[r], m.k11[r] * thick[r])
    t2 = np.where(vert, m.k33[c], m.k11[c] * thick[c])
    cond = np.where(vert, w / (0.5 * thick[r] / m.k33[r] + 0.5 * thick[c] / m.k33[c]),
                    w * t1 * t2 / (t1 * l2 + t2 * l1))
    chd = np.zeros(n, bool)
    chd[m.chd_node] = True
    head = m.strt.copy()
    head[m.chd_node] = m.chd_head
    rhs = np.zeros(n)
    np.add.at(rhs, m.wel_node, -m.wel_q)
    np.add.at(rhs, m.rch_node, -m.rch_rate * m.area[m.rch_node])
    amat = np.zeros(ja.size)
    amat[ia[:-1]] = -np.bincount(r, weights=cond, minlength=n)
    v = np.where(chd[r] | chd[c], 0.0, cond)
    e = ~chd[r] & chd[c]
    np.subtract.at(rhs, r[e], cond[e] * head[c[e]])
    amat[off] = v
    amat[ia[:-1][chd]] = 1.0
    rhs[chd] = head[chd]
    return ia, ja, amat, rhs, head


def _network64(p, ia, ja, amat, x, t, mask, inv, train):
    """The network in 64 bits: hidden 64, 8 message-passing layers over the
    symmetrically normalised off-diagonal entries, a linear read-out."""
    n = ia.size - 1
    row = np.repeat(np.arange(n), np.diff(ia))
    c = np.where(row == ja, 0.0, np.maximum(-amat, 0.0))
    deg = np.bincount(row, weights=c, minlength=n)
    dd = deg[row] * deg[ja]
    w = np.where(dd > 0, c / np.sqrt(np.where(dd > 0, dd, 1.0)), 0.0)
    s = torch.sparse_csr_tensor(torch.from_numpy(ia.astype(np.int64)), torch.from_numpy(ja.astype(np.int64)),
                                torch.from_numpy(w), size=(n, n)).to(DEV)
    q = torch.from_numpy(p.astype(np.float64)).to(DEV).requires_grad_(train)

    class Product(torch.autograd.Function):
        @staticmethod
        def forward(ctx, h):
            return s @ h

        @staticmethod
        def backward(ctx, g):  # the matrix is symmetric
            return s @ g

    sizes = [16 * 64, 64] + [128 * 64, 64] * 8 + [64, 1]
    part = list(torch.split(q, sizes))
    h = torch.relu(torch.from_numpy(x.astype(np.float64)).to(DEV) @ part[0].view(16, 64) + part[1])
    for l in range(8):
        z = torch.cat([h, Product.apply(h)], dim=1) @ part[2 + 2 * l].view(128, 64) + part[3 + 2 * l]
        h = h + torch.relu(z)
    y = h @ part[-2] + part[-1]
    if not train:
        return y.detach()
    e = (y - torch.from_numpy(t.astype(np.float64)).to(DEV)) * torch.from_numpy(mask.astype(np.float64)).to(DEV)
    loss = (e * e).sum() * inv
    loss.backward()
    return dict(loss=np.float32(float(loss.detach())), gradient=q.grad.detach().cpu().numpy())


def exact(case, seed):
    if case["kind"] == "gwf":
        if case["grid"] in ("newton", "xt3d") or case["nlay"] * case["nrow"] * case["ncol"] > 1_000_000:
            return None
        m = _model(case, seed)
        return _solve64(*(_system(m) if case["grid"] == "dis" else _grid_system(m))).cpu().numpy()
    if case["kind"] == "linear":
        m = _dis_model(case["nlay"], case["nrow"], case["ncol"], seed)
        x = _solve64(*_system(m))
        return x.cpu().numpy() if case["host"] else x
    if case["kind"] == "ensemble":
        return _solve64(*_concat([_system(m) for m in _ensemble_models(case, seed)])[1:])
    m, ia, ja, amat, p, x, t, mask = _network_inputs(case, seed)
    return _network64(p, ia, ja, amat, x, t, mask, 1.0 / float(mask.sum()), case["train"])
