"""Projection onto and synthesis from an installed basis at the edges of their tiling: one trajectory, remainders of the
trajectories that share a row's cells, one row to 64, the smallest and the largest grid of the batched ground states."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(8, 8, 64), (16, 16, 128), (32, 32, 256)])
@pytest.mark.parametrize("n,rows", [(1, 64), (5, 17), (9, 1)])
def test_projection_and_synthesis(grid, n, rows):
    cells = int(np.prod(grid))
    rng = np.random.default_rng(n)
    basis = np.linalg.qr(rng.normal(size=(cells, rows)))[0].T.astype(np.float32)
    coef_in = np.zeros((n, 64))
    coef_in[:, :rows] = rng.normal(size=(n, rows))
    groups = [rb87_params(N=20000 + 2000 * i, grid=grid) for i in range(n)]
    with Engine(groups) as eng:
        eng.set_warmstart_basis(grid, np.ascontiguousarray(basis))
        coef, prof, _ = eng.ground_state_coeffs(max_steps=2, coef_in=coef_in, want_profiles=True)
        # FP32 sums of sixteen products a thread, of a warp, then FP64: 32 roundings of 6e-8 at most
        B = basis.astype(np.float64)
        want = np.linalg.solve(B @ B.T, B @ prof.reshape(n, cells).astype(np.float64).T).T
        scale = np.linalg.norm(prof.reshape(n, cells), axis=1, keepdims=True)
        assert (np.abs(coef[:, :rows] - want) <= 2e-6 * scale).all()
        assert not coef[:, rows:].any()
        # the evolution's buffers hold the states before an ensemble is initialised, a workspace after: the same states
        eng.init_groups(range(n), [np.full(cells, 3.0)] * n)
        again = eng.ground_state_coeffs(max_steps=2, coef_in=coef_in, want_profiles=True)[1]
    # trajectories share nothing: each alone gives what the batch gives, up to the last bit of its norm
    np.testing.assert_allclose(again, prof, rtol=0, atol=1e-6)
    for t in (0, n - 1):
        with Engine(groups[t:t + 1]) as one:
            one.set_warmstart_basis(grid, np.ascontiguousarray(basis))
            alone = one.ground_state_coeffs(max_steps=2, coef_in=coef_in[t:t + 1], want_profiles=True)[1]
        np.testing.assert_allclose(alone[0], prof[t], rtol=0, atol=1e-6)
