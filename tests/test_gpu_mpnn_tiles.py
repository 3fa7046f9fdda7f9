"""The network's gradients at the sizes where their launches change: part of a
tile of 32 nodes, one tile and one node more, 148 tiles (the last size whose
kernels overlap) and one more, one tile per CTA (296) and one more.  Only the
first and the last three nodes miss their targets, by 100, so that what an
edge drops or counts twice shows; against the network's FP64 oracle at its bar
(1e-2 of a parameter group's largest entry)."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import learned as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 148 * 32, 148 * 32 + 1, 296 * 32, 296 * 32 + 1])
def test_gradients_match_oracle(n):
    import mpnn_oracle as O

    rng = np.random.default_rng(n)
    nbr = rng.integers(0, n, size=(n, 8))
    nbr[rng.random((n, 8)) < 0.2] = -1
    x = rng.normal(size=(n, L.IN)).astype(np.float32)
    w = L.init_weights(7)
    w[-(6 * 64 + 6):] = rng.normal(scale=0.1, size=6 * 64 + 6)
    net = L.MPNN(n, w)
    net.set_graph(torch.from_numpy(nbr.astype(np.int32)).cuda())
    xd = torch.from_numpy(x).cuda()
    y = net.forward(xd).cpu().numpy().reshape(n, L.OUT).copy()
    for i in {0, max(n - 3, 0), max(n - 2, 0), n - 1}:
        y[i] += rng.choice([-100.0, 100.0], L.OUT).astype(np.float32)
    loss, g = net.gradients(xd, torch.from_numpy(y).cuda())
    loss_o, g_o = O.loss_and_grad(w.astype(np.float64), x, y, nbr)
    assert abs(loss - loss_o) / loss_o < 1e-4
    o = 0
    for name, shp in O.SHAPES:
        k = int(np.prod(shp))
        a, b = g[o:o + k], g_o[o:o + k]
        assert np.abs(a - b).max() <= 1e-2 * max(np.abs(b).max(), 1e-12), name
        o += k
