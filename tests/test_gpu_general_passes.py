"""The general FP32 passes (planes that are not 8, 16 or 32 square, other nz, 2D slices) at the edges of their tiling,
against the CPU oracle: 2-point axes, every remainder of three stages per barrier, one and several planes per CTA, two to
sixteen pencils per CTA, the longest pencils and the largest planes; and the two sources of the kinetic phases."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [((2, 4, 8), 3), ((4, 1, 2), 1), ((64, 1, 64), 2), ((16, 4, 16), 5), ((8, 8, 32), 2), ((2, 2, 512), 1), ((64, 32, 4), 1),
         ((32, 64, 2), 1), ((2, 1024, 4), 1), ((1024, 1, 8), 1), ((32, 1, 128), 150)]


@pytest.mark.parametrize("grid,ne", GRIDS)
@pytest.mark.parametrize("itmax", [1, 3])
def test_steps_samples_and_pulses(grid, ne, itmax):
    p = rb87_params(N=20000, grid=grid, ne=ne, noise=True, seed=9, itmax=itmax)
    cells = int(np.prod(grid))
    rng = np.random.default_rng(1)
    gs = np.sqrt(20000.0 / (cells * O.derive(p).dV)) * (1.0 + 0.2 * rng.normal(size=cells))
    ref = O.OracleEnsemble(p)
    ref.init(gs)
    ref.start_evolution()
    with Engine([p], path=BEC_PATH_FP32_BATCHED) as eng:
        eng.init_group(0, gs)
        eng.start_evolution()
        mom, ax = eng.run(12, sample_every=6, pi_pulse_step=6, axial=True)
        ref.evolve(6)
        m1 = ref.moments()
        ref.pulse(np.pi)
        ref.evolve(6)
        for got, want in ((mom[0, 0], m1), (mom[1, 0], ref.moments())):
            np.testing.assert_allclose(got[1:], want[1:], rtol=0, atol=1e-4 * want[1:3].max())
        np.testing.assert_allclose(ax[0][1], ref.axial(), rtol=0, atol=1e-4 * np.abs(ref.axial()).max())
        # single precision over a dozen steps; the bound of the other state comparisons
        for t in range(min(ne, 3)):
            a, b = eng.get_state(0, t), ref.get_state(t)
            assert np.abs(a - b).max() < 2e-4 * np.abs(b).max()


def test_phases_from_the_table_and_in_place_are_the_same():
    """Above 256 MiB of tables the z pass evaluates the phases itself: the same bits."""
    grid, n = (64, 32, 16), 520
    groups = [rb87_params(N=20000 + 10 * i, grid=grid, noise=True, seed=i) for i in range(n)]
    cells = int(np.prod(grid))
    gs = (30.0 + np.random.default_rng(2).normal(size=cells)).astype(np.float32)
    states = []
    for some in (groups, groups[:1]):
        with Engine(some, path=BEC_PATH_FP32_BATCHED) as eng:
            eng.init_groups(range(len(some)), [gs] * len(some))
            eng.start_evolution()
            eng.run(4, sample_every=2, axial=True)
            states.append(eng.get_state(0, 0))
    np.testing.assert_array_equal(states[0], states[1])
