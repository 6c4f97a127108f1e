"""The packets of an unpeeled run in the two kernels it has: the tallies are
the same integers whether nearly every event runs in the lanes of the batch
kernel or, a warp per packet, in the one that takes what it leaves."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,prec,n", [
    ("tiny", hc3d.PREC_MIXED, 6000), ("tiny3d", hc3d.PREC_MIXED, 6000), ("tiny_acc", hc3d.PREC_MIXED, 3000),
    ("tiny_sg", hc3d.PREC_MIXED, 4000), ("tiny_isrf", hc3d.PREC_MIXED, 6000), ("plain", hc3d.PREC_MIXED, 6000),
    ("tiny", hc3d.PREC_FP64, 3000), ("tiny3d", hc3d.PREC_FP64, 3000), ("tiny_sg", hc3d.PREC_FP64, 2000)])
def test_both_kernels_give_the_same_tallies(tmp_path, built, name, prec, n):
    """One block of four warps takes hundreds of packets a lane and leaves at
    most 15 a warp; the default launch spreads as many packets over all
    warps, one or two lanes each, which all leave theirs at once."""
    m = make_model(tmp_path, name, MAXINT=2000)
    p = m.run_params(np=n, iter=1 if m.sg else 3, ipeel=0)
    got = []
    for blocks in (1, 0):
        ctx = hc3d.Context(prec, grid_blocks=blocks).load(m)
        ctx.zero()
        ctx.run(p)
        got.append(ctx.tallies(p))
        ctx.close()
    assert got[0]["counters"][hc3d.CNT["events"]] > n
    for key, v in got[0].items():
        if isinstance(v, np.ndarray):
            np.testing.assert_array_equal(v, got[1][key], err_msg=key)
