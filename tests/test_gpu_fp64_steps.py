"""The FP64 path's fused real-time passes at the edges of their tiling, against the CPU oracle: 2-point axes, every
remainder of radix 8, several planes per CTA, one to eight pencils, the largest plane of both components that fits in
shared memory, and one that does not (one kernel per operation)."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP64_PLAIN, Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-10     # the FP64 path's bar in the other parity tests

GRIDS = [((2, 1, 2), 1), ((4, 2, 8), 3), ((16, 16, 4), 40), ((32, 1, 16), 2), ((64, 64, 2), 1), ((128, 64, 2), 2), ((1024, 1, 4), 1),
         ((8, 8, 512), 1), ((2, 4, 1024), 1)]


def start(p):
    cells = p.nvx * p.nvy * p.nvz
    rng = np.random.default_rng(1)
    return np.sqrt(p.N / (cells * O.derive(p).dV)) * (1.0 + 0.2 * rng.normal(size=cells)) * np.exp(1j * rng.normal(size=cells))


@pytest.mark.parametrize("grid,ne", GRIDS)
@pytest.mark.parametrize("noise", [False, True])
def test_steps_samples_and_pulses(grid, ne, noise):
    p = rb87_params(N=20000, grid=grid, ne=ne, noise=noise, seed=9)
    gs = start(p)
    ref = O.OracleEnsemble(p)
    ref.init(gs)
    ref.start_evolution()
    with Engine([p], path=BEC_PATH_FP64_PLAIN) as eng:
        eng.init_group(0, gs)
        eng.start_evolution()
        mom, ax = eng.run(7, sample_every=3, pi_pulse_step=5, axial=True)
        ref.evolve(3)
        m1 = ref.moments()
        ref.evolve(2)
        ref.pulse(np.pi)
        ref.evolve(1)
        for got, want in ((mom[0, 0], m1), (mom[1, 0], ref.moments())):
            np.testing.assert_allclose(got[1:], want[1:], rtol=0, atol=TOL * want[1:3].max())
        np.testing.assert_allclose(ax[0][1], ref.axial(), rtol=0, atol=TOL * np.abs(ref.axial()).max())
        ref.evolve(1)
        for t in (0, ne - 1):
            a, b = eng.get_state(0, t), ref.get_state(t)
            assert np.abs(a - b).max() < TOL * np.abs(b).max()
            eng.set_state(0, t, a)
            assert np.abs(eng.get_state(0, t) - a).max() < 1e-14 * np.abs(a).max()


def test_a_run_has_the_same_bits_however_it_is_cut():
    p = rb87_params(N=20000, grid=(16, 8, 32), ne=3, noise=True, seed=4)
    gs, out = start(p), []
    for cuts in ((6,), (1, 3, 2)):
        with Engine([p], path=BEC_PATH_FP64_PLAIN) as eng:
            eng.init_group(0, gs)
            eng.start_evolution()
            for n in cuts:
                eng.evolve(n)
            out.append(eng.get_state(0, 2))
    np.testing.assert_array_equal(out[0], out[1])


def test_observation_in_several_parts():
    """More cells than one observation copies at once: the moments of every part."""
    p = rb87_params(N=20000, grid=(32, 32, 64), ne=35, noise=True, seed=4)
    with Engine([p], path=BEC_PATH_FP64_PLAIN) as eng:
        eng.init_group(0, start(p))
        eng.start_evolution()
        m = eng.run(1)[0, 0]
        na = sum((np.abs(eng.get_state(0, t)[0]) ** 2).sum() for t in range(35)) * O.derive(p).dV
    assert abs(m[1] - na) < 1e-12 * na
