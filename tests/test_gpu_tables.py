"""The Lucy CDF of the mixed form for table sizes on and off the tiles that the
device interleaves and searches it in: the mixed walk follows the FP64 form,
which reads the tables as they were given."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model, splitmix_uniforms, trace_key

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step_t,step_nu", [(27, 16), (333, 32), (9, 8), (3, 1), (111, 64)])
def test_thinned_tables(tmp_path, built, step_t, step_nu):
    """Every step_t-th of 1000 temperatures and step_nu-th of 1025 frequencies:
    (38,65), (4,33), (112,129), (334,1025), (10,17) rows and columns.  As many
    packets as with the whole tables take the same path in both forms."""
    m = make_model(tmp_path, "tiny")
    it, iu = np.arange(0, m.nT, step_t), np.arange(0, m.nnu, step_nu)
    nd = m.ndg_tab
    K = np.asarray(m.kapBint).reshape(m.nT, m.nnu, nd, order="F")[it][:, iu]
    kp = np.asarray(m.kappap).reshape(m.nT, nd, order="F")[it]
    m.lTint, m.nuint = np.ascontiguousarray(m.lTint[it]), np.ascontiguousarray(m.nuint[iu])
    m.kapBint, m.kappap = np.ravel(K, order="F").copy(), np.ravel(kp, order="F").copy()
    m.nT, m.nnu = len(it), len(iu)
    p = m.run_params(np=48, iter=3, ipeel=0)
    U = splitmix_uniforms(48, 8192, seed=3)
    got = [hc3d.Context(prec).load(m).trace(p, U, max_rec=2048) for prec in (hc3d.PREC_FP64, hc3d.PREC_MIXED)]
    keys = [[trace_key(r) for r in t] for t in got]
    assert sum(a.shape == b.shape and np.array_equal(a, b) for a, b in zip(*keys)) >= 0.75 * 48
