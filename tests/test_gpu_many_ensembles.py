"""Contexts of more ensembles than a grid's second dimension counts, on a grid of the general passes."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine

pytestmark = pytest.mark.gpu

GRID, N = (8, 1, 16), 70000


def test_seventy_thousand_ensembles_on_a_general_grid():
    few = [0, 1, 65535, 65536, N - 1]
    params = [rb87_params(N=20000 + g % 1000, grid=GRID, ne=1, noise=True, seed=g) for g in range(N)]
    gs = np.full(int(np.prod(GRID)), 30.0, dtype=np.float32)
    out = []
    for chosen in (range(N), few):
        with Engine([params[g] for g in chosen], path=BEC_PATH_FP32_BATCHED) as eng:
            eng.init_groups(range(eng.n_groups), [gs] * eng.n_groups)
            eng.start_evolution()
            eng.evolve(3)
            at = few if len(chosen) == N else range(len(few))
            out.append((np.stack([eng.get_state(g, 0) for g in at]), eng.moments()[list(at)]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
