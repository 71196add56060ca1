"""The warm-start network's kernels where each block walks several tiles of 64
nodes and the last tile is ragged, against the numpy restatement, with the
bounds of the small graphs (test_gpu_network.py); predictions and gradients in
turn on one handle."""
from types import SimpleNamespace

import numpy as np
import pytest

import mpnn_oracle
from modflow6_gb300.warmstart import WarmStartNet
from test_gpu_network import graph

pytestmark = pytest.mark.gpu


def test_several_tiles_a_block(gblib):
    import torch
    # two to three tiles a block forward (at most 608 blocks), four backward
    # (303), two and three for the input layer (1216 and 607); one node in the
    # last tile
    n = 80001
    ia, ja, amat = graph(n, 150, seed=3)
    net = WarmStartNet(SimpleNamespace(m=SimpleNamespace(nodes=n), nja=ja.size, ia=ia, ja=ja), seed=1)
    rng = np.random.default_rng(1)
    p = (rng.standard_normal(net.nparams) * 0.12).astype(np.float32)
    net.params = p
    dev = lambda a: torch.from_numpy(a).cuda()
    d_amat = dev(amat)
    net.set_graph(d_amat)
    x = rng.standard_normal((n, 16)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    mask = (rng.uniform(size=n) < 0.8).astype(np.float32)
    w = mpnn_oracle.edge_weights(ia, ja, amat)
    lo, go, yo = mpnn_oracle.loss_and_grad(p, ia, ja, w, x, t, mask, 1.0 / mask.sum())
    dx, dt, dm, inv = dev(x), dev(t), dev(mask), 1.0 / float(mask.sum())
    y = net.predict(dx).cpu().numpy()
    assert np.linalg.norm(y - yo) <= 5e-3 * np.linalg.norm(yo)
    # no tile stands out: each within four times that bound
    rms = np.sqrt(np.mean(yo**2))
    for r in range(0, n, 64):
        assert np.sqrt(np.mean((y[r:r + 64] - yo[r:r + 64]) ** 2)) <= 2e-2 * rms, r
    loss, g = net.gradients(dx, dt, dm, inv)
    assert abs(loss - lo) <= 5e-3 * lo
    assert np.linalg.norm(g - go) <= 2e-2 * np.linalg.norm(go)
    for name, part in (("W0", slice(0, 1024)), ("b0", slice(1024, 1088)), ("rest", slice(1088, None))):
        assert np.linalg.norm(g[part] - go[part]) <= 2e-2 * np.linalg.norm(go[part]), name
    # a prediction between two gradients, and after them: the same numbers (the
    # gradients but for the order of the atomic sums)
    np.testing.assert_array_equal(net.predict(dx).cpu().numpy(), y)
    loss2, g2 = net.gradients(dx, dt, dm, inv)
    assert loss2 == loss and np.linalg.norm(g2 - g) <= 1e-5 * np.linalg.norm(g)
    np.testing.assert_array_equal(net.predict(dx).cpu().numpy(), y)
    net.close()
