"""The report of the schedule for a context of many grid classes: whole for the Python engine, and in a buffer that held it
before the passes with four cells per thread were in it, without their fields."""
import ctypes as C
import json

import numpy as np
import pytest

from bec_b200.configs import rb87_params
from bec_b200.engine import BEC_PATH_FP32_BATCHED, Engine, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes", [3, 14, 20])
def test_report_fits(classes):
    grids = [(x, y, z) for z in (64, 128, 256) for x, y in ((8, 8), (16, 16), (32, 32), (16, 8), (8, 16), (32, 8), (4, 4))][:classes]
    with Engine([rb87_params(N=20000, grid=g, ne=1, noise=True, seed=1) for g in grids], path=BEC_PATH_FP32_BATCHED) as eng:
        for i, d in enumerate(eng.derived):
            eng.init_group(i, np.full(d.cells, 30.0))
        eng.start_evolution()
        whole = eng.step_plan
        assert [tuple(k["grid"]) for k in whole["pencil_kernels"]] == grids
        assert all("pair_ms" in k for k in whole["pencil_kernels"])
        buf = C.create_string_buffer(4096)
        assert lib().bec_step_plan(eng._h, buf, len(buf)) == 0
        small = json.loads(buf.value)
        if "pair_ms" not in small["pencil_kernels"][0]:
            for k in whole["pencil_kernels"]:
                for name in ("split_pencil", "split_plane", "pair_ms"):
                    del k[name]
        assert small == whole
