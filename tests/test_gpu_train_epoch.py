"""An epoch's minibatches in one launch, against Adam restated on the host with the
library's own gradient at each step's parameters: one, two and five minibatches of less
than a tile, several tiles with a ragged last one, a tile per block and more tiles than
blocks.

Tolerance, in units of the step size: an Adam step moves a parameter by lr m / sqrt(v),
whose FP32 rounding is led by 1 - 0.999^k (2^-24 / 0.001, halved by the root: 3e-5), and
the gradient of later steps differs by what those roundings of the parameters make of it;
1e-2 leaves that two orders of magnitude.  A tile, a row of sums or a wait left out
changes m / sqrt(v) of the second step on by a share of a minibatch, 1/700 of its sum at
the least and (five tiles) a fifth at the most, of its sign for many parameters.  The
loss is a mean of 0.5 e^2, each term with the rounding of two layers and the sums of the
gradient: 400 roundings of 2^-24."""
import numpy as np
import pytest

from pyclaw_b200.learned import Network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,steps", [(32, 1), (63, 5), (64, 2), (257, 5), (16384, 3), (44800, 2)])
def test_epoch_equals_steps(batch, steps):
    lr = np.float32(3e-3)
    net, ref = Network(seed=5), Network(seed=5)
    net.generate(batch * steps, seed=9)
    ref.generate(batch * steps, seed=9)
    P = ref.params.astype(np.float32)
    m, v, losses = np.zeros_like(P), np.zeros_like(P), []
    for k in range(steps):
        ref.params = P
        g, loss = ref.gradient(k * batch, batch)
        losses.append(loss)
        m = np.float32(0.9) * m + (np.float32(1) - np.float32(0.9)) * g
        v = np.float32(0.999) * v + (np.float32(1) - np.float32(0.999)) * g * g
        mh = m / (np.float32(1) - np.float32(0.9) ** np.float32(k + 1))
        vh = v / (np.float32(1) - np.float32(0.999) ** np.float32(k + 1))
        step = lr * (np.float32(1) - np.float32(0.9) * np.float32(k) / np.float32(steps))
        P = P - step * mh / (np.sqrt(vh) + np.float32(1e-8))
    last = net.train(1, batch, float(lr))
    assert np.abs(net.params - P).max() <= 1e-2 * lr
    assert abs(last - np.mean(losses)) <= 400 * 2.0 ** -24 * np.mean(losses)
    net.close()
    ref.close()
