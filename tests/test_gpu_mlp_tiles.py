"""The network's chain at the edges of its tiling against FP64: a single layer, widths and batches that are not multiples of
64, contractions of more stages than the ring holds, tiles of 16, 32 and 64 columns."""
import numpy as np
import pytest

from bec_b200.engine import MLP

pytestmark = pytest.mark.gpu

CASES = [((4, 3), 65), ((3, 40, 1), 20), ((5, 70, 130, 3), 100), ((6, 256, 64), 700), ((6, 512, 512, 64), 1000)]


def reference(widths, params, x, t):
    """Outputs, loss and gradients in FP64; params in the layout of get_params."""
    Ws, k = [], 0
    for a, b in zip(widths[:-1], widths[1:]):
        W = params[k:k + a * b].reshape(b, a).astype(np.float64)
        Ws.append((W, params[k + a * b:k + a * b + b].astype(np.float64)))
        k += a * b + b
    acts = [x.astype(np.float64)]
    for i, (W, b) in enumerate(Ws):
        z = acts[-1] @ W.T + b
        acts.append(np.tanh(z) if i < len(Ws) - 1 else z)
    d = 2.0 * (acts[-1] - t) / acts[-1].size
    grads = []
    for i in range(len(Ws) - 1, -1, -1):
        grads = [(d.T @ acts[i]).ravel(), d.sum(0)] + grads
        if i:
            d = (d @ Ws[i][0]) * (1.0 - acts[i] ** 2)
    return acts[-1], ((acts[-1] - t) ** 2).mean(), np.concatenate(grads)


@pytest.mark.parametrize("widths,batch", CASES)
def test_outputs_gradients_and_training(widths, batch):
    rng = np.random.default_rng(batch)
    x = rng.uniform(-1.0, 1.0, (batch, widths[0])).astype(np.float32)
    t = rng.normal(size=(batch, widths[-1])).astype(np.float32)
    with_bias = []
    for a, b in zip(widths[:-1], widths[1:]):
        with_bias += [rng.uniform(-1, 1, a * b) * np.sqrt(3.0 / a), rng.normal(0, 0.05, b)]
    p = np.concatenate(with_bias).astype(np.float32)
    net = MLP(widths, seed=1)
    try:
        net.set_params(p)
        y, loss, grads = reference(widths, p, x, t)
        # two BF16 values hold 16 bits of an operand: products off by 2 x 2^-17, sums of 512 of them by less than 1e-4 of
        # the largest after four layers
        assert np.abs(net.forward(x) - y).max() < 1e-4 * np.abs(y).max()
        got_loss, got = net.gradients(x, t)
        assert abs(got_loss - loss) < 1e-4 * loss
        assert np.abs(got - grads).max() < 1e-4 * np.abs(grads).max()
        # the whole set as one minibatch: its loss does not depend on the order of the draws
        hist = net.train(x, t, 3, batch=batch, lr=1e-3, seed=2)
        assert abs(hist[0] - loss) < 1e-4 * loss
        want = reference(widths, net.get_params(), x, t)
        assert abs(net.gradients(x, t)[0] - want[1]) < 1e-4 * want[1] and want[1] < hist[0]
    finally:
        net.close()
