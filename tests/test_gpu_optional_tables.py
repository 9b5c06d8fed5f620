"""A byte limit under which a context can be made, initialised and stepped without the optional tables of the general passes:
they are given up, and the run has the same bits."""
import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, BecError, Engine

pytestmark = pytest.mark.gpu

GRID, N = (4, 4, 512), 8          # state, staging area and tables: 1 MiB each


def run(params, monkeypatch, limit=None):
    if limit:
        monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(limit))
    with Engine(params, path=BEC_PATH_FP32_BATCHED) as eng:
        monkeypatch.delenv("BEC_DEVICE_BYTES_LIMIT", raising=False)
        eng.init_groups(range(N), [np.full(int(np.prod(GRID)), 30.0, dtype=np.complex128)] * N)
        eng.start_evolution()
        eng.evolve(4)
        return np.stack([eng.get_state(g, 0) for g in range(N)])


def smallest(params, monkeypatch, step=1 << 16):
    """The smallest limit, to 64 KiB, that creation passes."""
    bare = step
    while True:
        monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(bare))
        try:
            Engine(params, path=BEC_PATH_FP32_BATCHED).close()
            break
        except BecError:
            bare += step
    monkeypatch.delenv("BEC_DEVICE_BYTES_LIMIT")
    return bare


def test_tables_leave_room_for_the_initialisation(monkeypatch):
    params = [rb87_params(N=20000 + g, grid=GRID, ne=1, noise=True, seed=g) for g in range(N)]
    bare = smallest(params, monkeypatch)
    want = run(params, monkeypatch)
    for extra in (2, 8, 15, 16, 17, 24, 40):         # 64 KiB each, beside the staging area
        got = run(params, monkeypatch, bare + (1 << 20) + (extra << 16))
        np.testing.assert_array_equal(got, want)


def test_tables_given_back_while_steps_are_captured(monkeypatch):
    """The states come one by one, so that the staging area is first asked for when captured steps read the tables."""
    params = [rb87_params(N=20000 + g, grid=GRID, ne=1, noise=True, seed=g) for g in range(N)]
    cells = int(np.prod(GRID))
    out = []
    for bounded in (False, True):          # room for the tables or the staging area, not for both
        if bounded:
            monkeypatch.setenv("BEC_DEVICE_BYTES_LIMIT", str(smallest(params, monkeypatch) + (1 << 20) + (1 << 18)))
        with Engine(params, path=BEC_PATH_FP32_BATCHED) as eng:
            monkeypatch.delenv("BEC_DEVICE_BYTES_LIMIT", raising=False)
            for g in range(N):
                eng.set_state(g, 0, np.full(2 * cells, 30.0 + g, dtype=np.complex128))
            eng.evolve(40)
            eng.init_group(2, np.full(cells, 30.0, dtype=np.complex128))
            eng.evolve(40)
            out.append(np.stack([eng.get_state(g, 0) for g in range(N)]))
    np.testing.assert_array_equal(out[0], out[1])
