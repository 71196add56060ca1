"""The warm-start network's layer kernels (k_mpnn.cu) on graphs at the edges
of their tiles (64 nodes) and of a gather's first 8 neighbours, against the
numpy restatement with the same BF16 operand rounding: only the order of FP32
sums differs (1e-6 or so), and where that flips a BF16 rounding (2^-9 of one
operand out of 128) the outputs move by well under 5e-3 of their norm."""
from types import SimpleNamespace

import numpy as np
import pytest

import mpnn_oracle
from modflow6_gb300.warmstart import WarmStartNet

pytestmark = pytest.mark.gpu


def graph(n, hub, seed):
    """A ring with random chords, and one node joined to `hub` others."""
    rng = np.random.default_rng(seed)
    nb = [set() for _ in range(n)]
    pairs = [(i, i + 1) for i in range(n - 1)] + [(0, j) for j in range(1, min(n, hub + 1))]
    pairs += [tuple(rng.choice(n, 2, replace=False)) for _ in range(n if n > 2 else 0)]
    for i, j in pairs:
        nb[i].add(j)
        nb[j].add(i)
    ia = np.cumsum([0] + [1 + len(s) for s in nb]).astype(np.int32)
    ja = np.concatenate([[i] + sorted(s) for i, s in enumerate(nb)]).astype(np.int32)
    c = {}
    amat = np.zeros(ja.size)
    for i in range(n):
        for p in range(ia[i] + 1, ia[i + 1]):
            k = (min(i, ja[p]), max(i, ja[p]))
            amat[p] = c.setdefault(k, rng.uniform(0.1, 2.0)) * -1.0
    return ia, ja, amat


@pytest.mark.parametrize("n,hub", [(1, 0), (2, 0), (63, 8), (64, 9), (65, 16), (200, 150)])
def test_layers_match_numpy(gblib, n, hub):
    import torch
    ia, ja, amat = graph(n, hub, seed=n)
    net = WarmStartNet(SimpleNamespace(m=SimpleNamespace(nodes=n), nja=ja.size, ia=ia, ja=ja), seed=1)
    rng = np.random.default_rng(n + 1)
    p = (rng.standard_normal(net.nparams) * 0.12).astype(np.float32)
    net.params = p
    dev = lambda a: torch.from_numpy(a).cuda()
    d_amat = dev(amat)
    net.set_graph(d_amat)
    x = rng.standard_normal((n, 16)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    mask = (rng.uniform(size=n) < 0.8).astype(np.float32)
    mask[0] = 1.0
    w = mpnn_oracle.edge_weights(ia, ja, amat)
    lo, go, yo = mpnn_oracle.loss_and_grad(p, ia, ja, w, x, t, mask, 1.0 / mask.sum())
    y = net.predict(dev(x)).cpu().numpy()
    assert np.linalg.norm(y - yo) <= 5e-3 * np.linalg.norm(yo)
    loss, g = net.gradients(dev(x), dev(t), dev(mask), 1.0 / float(mask.sum()))
    assert abs(loss - lo) <= 5e-3 * lo
    assert np.linalg.norm(g - go) <= 2e-2 * np.linalg.norm(go)
    # a forward pass without a target leaves the gradients' buffers alone
    loss2, g2 = net.gradients(dev(x), dev(t), dev(mask), 1.0 / float(mask.sum()))
    assert abs(loss2 - loss) == 0.0 and np.linalg.norm(g2 - g) <= 1e-5 * np.linalg.norm(g)
    net.close()
