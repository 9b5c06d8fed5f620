"""Captured stretches of steps, a chain of launches per grid class: the same bits as launching every kernel, for a context
with more classes than streams, for one of a single class, and for one whose chains run one after another; every stretch
length that takes another mix of the captured graphs."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu

TEN = [(8, 8, 64), (16, 16, 64), (32, 32, 64), (16, 8, 64), (8, 8, 32), (4, 4, 512), (32, 16, 16), (128, 1, 32), (32, 1, 128), (2, 2, 8)]
CONTEXTS = {
    "ten_classes": [rb87_params(N=20000 + 1000 * i, grid=g, ne=1 + i % 3, noise=True, seed=i) for i, g in enumerate(TEN)],
    "one_class": [rb87_params(N=20000, grid=(16, 16, 128), ne=3, noise=True, seed=4)],
    "large": [rb87_params(N=20000, grid=g, ne=ne, noise=True, seed=4) for g, ne in (((32, 32, 256), 60), ((16, 16, 64), 90))],
}


def states(groups, graphs, monkeypatch):
    monkeypatch.setenv("BEC_CUDA_GRAPHS", "1" if graphs else "0")
    with Engine(groups, path=BEC_PATH_FP32_BATCHED) as eng:
        for g, d in enumerate(eng.derived):
            eng.init_group(g, 30.0 + np.random.default_rng(g).normal(size=d.cells))
        eng.start_evolution()
        out = []
        for n in (2, 9, 75 if len(groups) != 2 else 12, 1):
            eng.evolve(n)
            out.append(np.concatenate([eng.get_state(g, p.ne - 1).reshape(-1) for g, p in enumerate(groups)]))
        return out


@pytest.mark.parametrize("name", CONTEXTS)
def test_captured_chains_have_the_bits_of_single_launches(name, monkeypatch):
    monkeypatch.setenv("BEC_STEP_PLAN", "unfused")
    got, want = (states(CONTEXTS[name], graphs, monkeypatch) for graphs in (True, False))
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
