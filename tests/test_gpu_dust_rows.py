"""Dust tables around the size that still fits in a block's shared memory
beside what the kernels keep there themselves."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.test_gpu_dust_files import _model

pytestmark = pytest.mark.gpu


# with the 241 rows of the other file: 1224, 1225 (49000 bytes in FP64), 1226, 1228 (49120), 1229 (49160 > 48 KB)
@pytest.mark.parametrize("rows", [983, 984, 985, 987, 988])
@pytest.mark.parametrize("ipeel", [0, 1])
def test_rows_at_the_limit_of_shared_memory(tmp_path, built, rows, ipeel):
    m = _model(tmp_path, rows)
    n = 500
    p = m.run_params(np=n, iter=3, ipeel=ipeel)
    ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
    ctx.zero()
    ctx.run(p)
    c = ctx.tallies(p)["counters"]
    ctx.close()
    assert c[hc3d.CNT["escaped"]] + c[hc3d.CNT["aflux"]] + c[hc3d.CNT["abflux"]] == n
    assert np.all(c >= 0)
