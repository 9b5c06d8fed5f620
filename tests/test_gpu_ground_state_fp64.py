"""bec_ground_state (FP64) against the CPU oracle at the edges of the fused passes' range: one- and two-point axes,
every remainder of the radix-8 stages (2^k points, k mod 3 = 0, 1, 2), several planes per CTA and one, tiles of two to
eight pencils, the largest plane that fits in shared memory, and a plane that does not (one kernel per operation)."""
import numpy as np
import pytest

from bec_b200._abi import BEC_GS_FIXED_STEPS, BEC_GS_MU, BEC_GS_MU_RESIDUAL, BEC_GS_REFERENCE_E
from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, BEC_PATH_FP64_PLAIN, Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(2, 1, 2), (4, 2, 8), (16, 1, 8), (32, 1, 128), (8, 8, 64), (16, 8, 64), (4, 4, 512), (64, 32, 16), (32, 32, 32),
         (128, 64, 4), (128, 128, 2), (8, 4, 1024)]
# the same FP64 arithmetic up to the order of sums and the factoring of exponentials: a few hundred roundings of
# 1.1e-16 per step and cell, 30 steps
TOL = 1e-11


def _path(grid):
    return BEC_PATH_FP64_PLAIN if grid[0] * grid[1] > 2048 or grid[2] > 512 else BEC_PATH_FP32_BATCHED


@pytest.mark.parametrize("grid", GRIDS)
def test_fixed_steps(grid):
    p = rb87_params(N=20000, grid=grid)
    # the points of a two-point axis lie outside the Thomas-Fermi profile, which is zero there: start from a given state
    warm = None if min(n for n in grid if n > 1) > 2 else 1.0 + np.random.default_rng(2).uniform(size=int(np.prod(grid)))
    kw = dict(mode=BEC_GS_FIXED_STEPS, max_steps=30, warm_start=warm)
    with Engine([p], path=_path(grid)) as eng:
        psi, rep = eng.ground_state(0, **kw)
        again, _ = eng.ground_state(0, **kw)
    ref, rr = O.ground_state(p, **kw)
    assert np.abs(psi - ref).max() < TOL * np.abs(ref).max()
    np.testing.assert_array_equal(psi, again)
    assert rep.steps == rr.steps == 30
    for k in ("mu", "energy", "N"):
        assert getattr(rep, k) == pytest.approx(getattr(rr, k), rel=TOL)
    assert rep.residual == pytest.approx(rr.residual, rel=1e-8, abs=1e-9)


@pytest.mark.parametrize("mode", [BEC_GS_MU, BEC_GS_MU_RESIDUAL, BEC_GS_REFERENCE_E])
@pytest.mark.parametrize("grid", [(8, 8, 64), (16, 8, 32), (32, 1, 128)])
def test_stopping_rules_and_warm_start(grid, mode):
    p = rb87_params(N=20000, grid=grid)
    kw = dict(mode=mode, max_steps=400, tol=1e-5, check_every=10, res_tol=1e-3)
    rng = np.random.default_rng(4)
    start, _ = O.ground_state(p, max_steps=5)
    start = start * (1.0 + 0.01j * rng.normal(size=start.size))     # a complex warm start stays complex
    for warm in (None, start):
        with Engine([p], path=BEC_PATH_FP64_PLAIN) as eng:
            psi, rep = eng.ground_state(0, warm_start=warm, **kw)
        ref, rr = O.ground_state(p, warm_start=warm, **kw)
        assert (rep.steps, rep.converged) == (rr.steps, rr.converged)
        assert np.abs(psi - ref).max() < TOL * np.abs(ref).max()
        assert rep.step_residual == pytest.approx(rr.step_residual, rel=1e-7)


def test_workspace_is_shared_by_grids_of_one_context():
    small, large = rb87_params(N=20000, grid=(8, 8, 64)), rb87_params(N=20000, grid=(16, 16, 64))
    with Engine([small, large], path=BEC_PATH_FP32_BATCHED) as eng:
        a, _ = eng.ground_state(0, max_steps=8)
        b, _ = eng.ground_state(1, max_steps=8, mode=BEC_GS_REFERENCE_E)
        c, _ = eng.ground_state(0, max_steps=8)
    np.testing.assert_array_equal(a, c)
    ref, _ = O.ground_state(large, max_steps=8, mode=BEC_GS_REFERENCE_E)
    assert np.abs(b - ref).max() < TOL * np.abs(ref).max()
