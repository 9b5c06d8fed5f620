"""Passes that the autotuner takes or leaves by their time, forced: four cells a thread in the pencil pass, the plane pass and
both, and the 8x8x64 step on-chip, against the wide passes, bit for bit; launched one by one and in captured stretches, whose
last plane launch advances the step index."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu

GRIDS = [(n, n, nz) for n in (8, 16, 32) for nz in (64, 128, 256)] + [(32, 1, 128), (16, 1, 256), (16, 8, 64)]
PLANS = {"unfused-split": (True, True), "unfused-split-pencil": (True, False), "unfused-split-plane": (False, True)}


def evolved(groups, plan, graphs, monkeypatch):
    monkeypatch.setenv("BEC_STEP_PLAN", plan)
    monkeypatch.setenv("BEC_CUDA_GRAPHS", "1" if graphs else "0")
    with Engine(groups, path=BEC_PATH_FP32_BATCHED) as eng:
        for g, d in enumerate(eng.derived):
            eng.init_group(g, 30.0 + np.random.default_rng(g).normal(size=d.cells))
        eng.start_evolution()
        eng.run(14, sample_every=5, pi_pulse_step=7)
        eng.evolve(43)                               # captured: 32 steps, 8 and single ones
        eng.evolve(3)
        states = np.concatenate([eng.get_state(g, t).reshape(-1) for g, p in enumerate(groups) for t in range(p.ne)])
        return states, eng.step_plan["pencil_kernels"]


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("grid", GRIDS)
def test_four_cells_a_thread(plan, grid, monkeypatch):
    groups = [rb87_params(N=20000, grid=grid, ne=3, noise=True, seed=7)]
    want, _ = evolved(groups, "unfused", False, monkeypatch)
    for graphs in (True, False):
        got, (kernels,) = evolved(groups, plan, graphs, monkeypatch)
        square = grid[0] == grid[1] and grid[0] < 32      # the planes that the split plane pass covers
        assert (kernels["split_pencil"], kernels["split_plane"]) == (PLANS[plan][0], PLANS[plan][1] and square)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("plan", ["unfused-split", "unfused-onchip"])
def test_chains_of_several_classes(plan, monkeypatch):
    grids = [(8, 8, 64), (16, 16, 64), (32, 32, 64), (16, 8, 64), (8, 8, 32), (32, 1, 128)]
    groups = [rb87_params(N=20000 + 1000 * i, grid=g, ne=1 + i % 3, noise=True, seed=i) for i, g in enumerate(grids)]
    want, _ = evolved(groups, "unfused", False, monkeypatch)
    for graphs in (True, False):
        got, kernels = evolved(groups, plan, graphs, monkeypatch)
        assert kernels[0]["onchip"] == (plan == "unfused-onchip")
        np.testing.assert_array_equal(got, want)
