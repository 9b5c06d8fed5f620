"""The passes with four cells a thread, which the autotuner may take for a class of few trajectories: the same bits as the
passes with sixteen, on every plane and pencil they cover, with a pulse and samples on the way."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu

GRIDS = [(n, n, nz) for n in (8, 16, 32) for nz in (64, 128, 256)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("ne", [1, 3])
def test_same_bits_as_the_wide_passes(grid, ne, monkeypatch):
    p = rb87_params(N=20000, grid=grid, ne=ne, noise=True, seed=7)
    gs = 30.0 + np.random.default_rng(0).normal(size=int(np.prod(grid)))
    out = []
    for plan in (None, "unfused"):
        monkeypatch.delenv("BEC_STEP_PLAN", raising=False)
        if plan:
            monkeypatch.setenv("BEC_STEP_PLAN", plan)
        with Engine([p], path=BEC_PATH_FP32_BATCHED) as eng:
            eng.init_group(0, gs)
            eng.start_evolution()
            eng.run(14, sample_every=5, pi_pulse_step=7)
            eng.evolve(3)
            out.append(np.concatenate([eng.get_state(0, t) for t in range(ne)]))
    np.testing.assert_array_equal(out[0], out[1])
