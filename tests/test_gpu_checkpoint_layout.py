"""The order of a cell inside a batched-path checkpoint: (a.re, a.im, b.re, b.im) per cell, trajectories by grid
class, whatever order the kernels keep a cell in. Files written by earlier builds stay loadable."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,ne", [((8, 8, 64), 3), ((16, 8, 32), 1), ((32, 1, 128), 2)])
def test_checkpoint_cell_order(grid, ne):
    nx, ny, nz = grid
    cells = nx * ny * nz
    p = rb87_params(N=20000, grid=grid, ne=ne, noise=True, seed=3)
    rng = np.random.default_rng(1)
    with Engine([p], path=BEC_PATH_FP32_BATCHED) as eng:
        eng.init_group(0, rng.normal(size=cells) + 1j * rng.normal(size=cells))
        eng.start_evolution()
        eng.evolve(3)
        states = [eng.get_state(0, t).reshape(2, nz, ny, nx) for t in range(ne)]   # x-space; ends the step
        blob = eng.checkpoint()
        # a payload cell (complex64 a, b) is the inverse transform over x and y, unnormalised, of the x-space state
        got = np.frombuffer(blob[-16 * cells * ne:], dtype=np.complex64).reshape(ne, nz, ny, nx, 2)
        for t in range(ne):
            for c in range(2):
                ref = np.fft.ifft2(states[t][c], axes=(1, 2)) * (nx * ny)
                # FP32 transforms of up to 1024 points on both sides: 1e-5 of the largest value covers them
                assert np.abs(got[t, ..., c] - ref).max() < 1e-5 * np.abs(ref).max()
        # the same bytes give the same run again
        m = eng.run(5, sample_every=5)
        with Engine([p], path=BEC_PATH_FP32_BATCHED) as other:
            other.restore(blob)
            np.testing.assert_array_equal(other.run(5, sample_every=5), m)
