"""Peel-off rays towards any number of directions, the one and the most that
are taken included: what one direction gets does not depend on the others."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n", [("tiny3d", 3), ("tiny3d", 256), ("tiny", 255)])
def test_each_direction_by_itself(tmp_path, built, name, n):
    th = ["%.3f" % (1.0 + 178.0 * (j + 0.37) / n) for j in range(n)]
    ph = ["%.1f" % (j * 47.0 % 360.0) for j in range(n)]

    def run(idx):
        m = make_model(tmp_path, name, MAXINT=300, NPEEL=len(idx), NXIMG=31,
                       THETE=",".join(th[j] for j in idx), PHIE=",".join(ph[j] for j in idx))
        ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
        p = m.run_params(np=300, iter=3, ipeel=1)
        p.seed = 11
        ctx.zero()
        ctx.run(p)
        t = ctx.tallies(p, grid=False)
        ctx.close()
        return t

    whole = run(range(n))
    c = hc3d.CNT
    assert whole["counters"][c["peels"]] > 0 and whole["counters"][c["peel_stuck"]] == 0
    for j in (0, n // 2, n - 1):
        one = run([j])
        for q in ("ti", "tq", "tu", "tv", "ti2", "numt"):
            np.testing.assert_array_equal(one[q][:, 0], whole[q][:, j], err_msg=q)
        np.testing.assert_array_equal(one["image_i"][0], whole["image_i"][j])
    assert whole["numt"].sum() > 0
