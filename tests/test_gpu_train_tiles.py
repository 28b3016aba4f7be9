"""The training kernel's tiling (64 samples a tile, at most four CTAs per SM,
each looping over its tiles): the gradient at counts around the edges of a
tile and past the one-tile-per-CTA range, against the FP64 reference, and the
same result on a second call (the sums are added in a fixed order).

Tolerance: FP32 rounding of sums of positive and negative terms.  A parameter's
sum passes at most 64 terms per tile, the CTA's tiles and the rows of partial
sums in sequence, and each term carries the rounding of the two layers (sums
of 32) and their tanh: 400 roundings of 2^-24 times the sum of the terms'
magnitudes."""
import numpy as np
import pytest

from oracle import mlp_ref as ref
from pyclaw_b200.learned import Network

pytestmark = pytest.mark.gpu


def _magnitude(P, x, y):
    """Largest sum of |terms| over the parameters, mean over the samples."""
    W1, b1, W2, b2, W3, b3 = ref.unpack(P)
    out, h1, h2 = ref.forward(P, x)
    dy = np.abs(out - y) / len(x)
    dz2 = dy[:, None] * np.abs(W3) * (1.0 - h2 ** 2)
    dz1 = (dz2 @ np.abs(W2)) * (1.0 - h1 ** 2)
    return max(dy.sum(), (np.abs(h2).T @ dy).max(), (dz2.T @ np.abs(h1)).max(), (dz1.T @ np.abs(x)).max(),
               dz1.sum(0).max())


@pytest.mark.parametrize("first,count", [(0, 1), (5, 63), (0, 64), (3, 65), (0, 128), (17, 40000), (0, 90001)])
def test_gradient_at_tile_edges(first, count):
    net = Network(seed=11)
    net.generate(first + count, seed=3)
    g, loss = net.gradient(first, count)
    again, loss2 = net.gradient(first, count)
    assert np.array_equal(g, again) and loss == loss2
    x8, y, ok = net.samples(first, count)
    on = ok != 0
    x, t = x8[on, :6].astype(np.float64), y[on].astype(np.float64)
    if not on.any():
        assert not g.any() and loss == 0.0
        return
    gr, lr = ref.gradient(net.params, x, t)
    share = on.sum() / count  # the mean runs over every sample, invalid ones adding nothing
    tol = 400 * 2.0 ** -24 * _magnitude(net.params, x, t) * share
    assert np.abs(g - gr * share).max() <= tol
    assert abs(loss - lr * share) <= 400 * 2.0 ** -24 * lr * share
    net.close()
