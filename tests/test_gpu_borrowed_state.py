"""A batch of ground states in a context without initialised ensembles works in the evolution's buffers: it leaves them as it
found them."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu


def test_unset_trajectories_stay_empty():
    """Of an ensemble of three, one state is set: the others are zero, with or without ground states before."""
    grid = (8, 8, 64)
    groups = [rb87_params(N=20000, grid=grid, ne=ne, noise=True, seed=ne) for ne in (3, 1)]
    state = np.full(2 * int(np.prod(grid)), 30.0, dtype=np.complex128)
    out = []
    for before in (False, True):
        with Engine(groups, path=BEC_PATH_FP32_BATCHED) as eng:
            if before:
                eng.ground_state_coeffs(groups=[0, 1], max_steps=5)
            eng.set_state(0, 1, state)
            eng.set_state(1, 0, state)
            out.append((eng.moments(), eng.get_state(0, 0), eng.get_state(0, 2)))
    assert not out[0][1].any() and not out[0][2].any()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
