"""A network whose call failed on the host's account: what later calls compute."""
import numpy as np
import pytest

from bec_b200.engine import MLP, BecError

pytestmark = pytest.mark.gpu

WIDTHS = (6, 130, 64)
LOSS = 1e-5         # a loss is a sum of 64 atomic FP32 adds in any order: 2 x 63 x 2^-24


def samples(n):
    rng = np.random.default_rng(n)
    return rng.uniform(-1, 1, (n, WIDTHS[0])).astype(np.float32), rng.normal(size=(n, WIDTHS[-1])).astype(np.float32)


@pytest.mark.parametrize("call", ["forward", "gradients", "train"])
@pytest.mark.parametrize("grown", [False, True])
def test_refused_batch_leaves_small_ones_as_they_were(call, grown, monkeypatch):
    small, more, large = samples(100), samples(1000), samples(200000)
    monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(1 << 25))       # 32 MiB: the large batch takes hundreds
    bounded = MLP(WIDTHS, seed=3)
    monkeypatch.delenv("BEC_DEVICE_BYTES_LIMIT")
    free = MLP(WIDTHS, seed=3)

    def use(net, x, t):
        if call == "forward":
            return net.forward(x)
        if call == "gradients":
            return net.gradients(x, t)[1]
        net.train(x, t, 3, batch=len(x))
        return net.get_params()

    if grown:                                   # the first batch's buffers are already replaced by larger ones
        np.testing.assert_array_equal(use(bounded, *more), use(free, *more))
    with pytest.raises(BecError, match="OUT_OF_MEMORY"):
        use(bounded, *large)
    np.testing.assert_array_equal(bounded.get_params(), free.get_params())
    np.testing.assert_array_equal(bounded.forward(small[0]), free.forward(small[0]))
    got, want = bounded.gradients(*small), free.gradients(*small)
    assert abs(got[0] - want[0]) < LOSS * want[0]
    np.testing.assert_array_equal(got[1], want[1])
    bounded.train(*small, 3, batch=64)
    free.train(*small, 3, batch=64)
    np.testing.assert_array_equal(bounded.get_params(), free.get_params())
    bounded.close()
    free.close()


@pytest.mark.parametrize("steps", [1, 2, 3])
def test_training_that_gave_up_leaves_operands_of_its_weights(steps, monkeypatch):
    x, t = samples(100)
    net, fresh = MLP(WIDTHS, seed=3), MLP(WIDTHS, seed=4)
    monkeypatch.setenv("BEC_GEMM_INJECT_STALL", "1")
    monkeypatch.setenv("BEC_STEP_WAIT_LIMIT_MS", "20")
    with pytest.raises(BecError):
        net.train(x, t, steps, batch=64)
    monkeypatch.delenv("BEC_GEMM_INJECT_STALL")
    monkeypatch.delenv("BEC_STEP_WAIT_LIMIT_MS")
    fresh.set_params(net.get_params())
    np.testing.assert_array_equal(net.forward(x), fresh.forward(x))
    got, want = net.gradients(x, t), fresh.gradients(x, t)
    np.testing.assert_allclose(got[0], want[0], rtol=LOSS)
    np.testing.assert_array_equal(got[1], want[1])
    net.close()
    fresh.close()
