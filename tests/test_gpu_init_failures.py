"""An initialisation that is refused (for want of memory, by the context's byte limit) on an evolving context: its steps go on
with the bits of a context that never asked."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, BecError, Engine

pytestmark = pytest.mark.gpu

GRID = (32, 32, 128)          # a ground state's staging area: 2 MiB


def params(groups):
    return [rb87_params(N=20000, grid=GRID, ne=1, noise=True, seed=g) for g in range(groups)]


def smallest_context(groups, monkeypatch, step=1 << 17):
    """The smallest byte limit (to `step` bytes) under which the context can be made, and the context."""
    limit = step
    while True:
        monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(limit))
        try:
            eng = Engine(groups, path=BEC_PATH_FP32_BATCHED)
        except BecError:
            limit += step
            continue
        eng.close()
        monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(limit + (1 << 19)))     # twiddles; no staging area
        eng = Engine(groups, path=BEC_PATH_FP32_BATCHED)
        monkeypatch.delenv("BEC_DEVICE_BYTES_LIMIT")
        return eng


@pytest.mark.parametrize("groups,pulse", [(1, False), (1, True), (2, False)])
def test_refused_initialisation_changes_nothing(groups, pulse, monkeypatch):
    rng = np.random.default_rng(groups)
    cells = int(np.prod(GRID))
    start = 30.0 + rng.normal(size=(groups, 2 * cells)) + 1j * rng.normal(size=(groups, 2 * cells))
    gs = [np.full(cells, 30.0, dtype=np.complex128) for _ in range(groups)]
    out = []
    for refuse in (False, True):
        eng = smallest_context(params(groups), monkeypatch) if refuse else Engine(params(groups), path=BEC_PATH_FP32_BATCHED)
        for g in range(groups):
            eng.set_state(g, 0, start[g])
        eng.evolve(5)                                    # its last half kick is due with the next step
        if pulse:
            eng.pulse(np.pi / 2)
        if refuse:
            with pytest.raises(BecError):
                eng.init_groups(range(groups), gs)
            if groups == 1:
                with pytest.raises(BecError):
                    eng.init_group(0, gs[0])
        eng.evolve(3)
        out.append(np.concatenate([eng.get_state(g, 0).reshape(-1) for g in range(groups)]))
        eng.close()
    np.testing.assert_array_equal(out[0], out[1])
