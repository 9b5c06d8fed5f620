"""The network at batches where a launch has more tiles than the chip has SMs and takes its widest ones: outputs, gradients and
trained parameters against FP64, with layers whose padded widths (64, 192) the widest tile does not divide."""
import numpy as np
import pytest

from bec_b200.engine import MLP
from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu

WARM = (6, 256, 256, 256, 64)


def network(widths, n):
    """A network with random parameters, the parameters, and n samples whose targets no network fits."""
    rng = np.random.default_rng(n)
    p = np.concatenate([v for a, b in zip(widths[:-1], widths[1:])
                        for v in (rng.uniform(-1, 1, a * b) * np.sqrt(3.0 / a), rng.normal(0, 0.05, b))]).astype(np.float32)
    net = MLP(widths, seed=1)
    net.set_params(p)
    return net, p, rng.uniform(-1, 1, (n, widths[0])).astype(np.float32), rng.normal(size=(n, widths[-1])).astype(np.float32)


# two BF16 values hold 16 bits of an operand: products off by 2 x 2^-17, sums of 512 of them by less than 1e-4 of the largest
# after four layers
@pytest.mark.parametrize("widths,rows", [(WARM, 9472), (WARM, 9473), (WARM, 20000), ((5, 70, 130, 3), 3137)])
def test_outputs(widths, rows):
    net, p, x, _ = network(widths, rows)
    y, want = net.forward(x), M.forward(p, widths, x)[-1]
    net.close()
    assert np.abs(y - want).max() < 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("widths,rows", [((5, 70, 130, 3), 3009), (WARM, 9473)])
def test_gradients(widths, rows):
    net, p, x, t = network(widths, rows)
    loss, grads = net.gradients(x, t)
    net.close()
    want_loss, want = M.loss_and_grads(p, widths, x, t)
    assert abs(loss - want_loss) < 1e-4 * want_loss
    assert np.abs(grads - want).max() < 1e-4 * np.abs(want).max()


@pytest.mark.parametrize("widths,n", [(WARM, 1088), (WARM, 1089), (WARM, 4096), ((6, 512, 512, 64), 1000), ((5, 70, 130, 3), 4096)])
def test_three_training_steps(widths, n):
    net, p, x, t = network(widths, n)
    lr = 1e-3
    net.train(x, t, 3, batch=n, lr=lr, seed=2)           # the whole set a step: the order of the draws does not matter
    got = net.get_params().astype(np.float64)
    net.close()
    want, m, v = p.astype(np.float64), 0.0, 0.0
    for s in range(1, 4):
        g = M.loss_and_grads(want, widths, x, t)[1]
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        want -= lr * (m / (1 - 0.9 ** s)) / (np.sqrt(v / (1 - 0.999 ** s)) + 1e-8)
    # An update is lr g / |g| at first, so a gradient's error counts by its size beside that gradient: e of a layer's typical
    # gradient, here 2^-15, moves the share of the layer's weights whose gradient is below e of it by up to 2 lr, and the others
    # by lr e / |g|: sqrt(5 e) lr in the mean square, 0.012 lr a step. A layer that is left out is 1 to 3 lr off.
    k = 0
    for a, b in zip(widths[:-1], widths[1:]):
        d = (got - want)[k:k + a * b + b]
        k += a * b + b
        assert np.sqrt((d * d).mean()) < 0.1 * lr, (a, b)
