"""The axial profile of an ensemble, summed on the device: around the sixteen loads in flight, and above and below the ensemble
from which a warp sums a value; beside a small ensemble that takes the same launch."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, BEC_PATH_FP64_PLAIN, Engine

pytestmark = pytest.mark.gpu


# FP64: sums of up to 4097 positive and mixed terms, compensated, of states read back in the same precision: 1e-12 of the
# largest covers both sides' rounding. FP32: the observing pass and the state's pass round a plane's 8 cells apart: 1e-5.
@pytest.mark.parametrize("path,tol", [(BEC_PATH_FP64_PLAIN, 1e-12), (BEC_PATH_FP32_BATCHED, 1e-5)])
@pytest.mark.parametrize("ne", [1, 15, 16, 17, 4096, 4097])
def test_profile_is_the_sum_over_the_trajectories(path, tol, ne):
    groups = [rb87_params(N=20000, grid=(4, 2, 4), ne=n, noise=True, seed=n) for n in (ne, 3)]
    with Engine(groups, path=path) as eng:
        for g, d in enumerate(eng.derived):
            eng.init_group(g, np.full(d.cells, 30.0, dtype=np.complex128))
        eng.start_evolution()
        mom, axial = eng.run(2, sample_every=2, axial=True)
        for g, d in enumerate(eng.derived):
            got = axial[g][0]
            np.testing.assert_allclose(got.sum(axis=0), mom[0, g, 1:], rtol=0, atol=1e-12 * mom[0, g, 1:3].max())
            want = np.zeros((d.nvz, 4))
            for t in range(groups[g].ne):
                a, b = eng.get_state(g, t).reshape(2, d.nvz, -1)
                c = (a.conj() * b).sum(axis=1)
                want += np.stack([(abs(a) ** 2).sum(axis=1), (abs(b) ** 2).sum(axis=1), c.real, c.imag], 1) * d.dV
            assert np.abs(got - want).max() < tol * want.max()
