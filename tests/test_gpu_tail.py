"""The packets that a batch leaves to the warp-per-packet kernel: a run's
tallies do not depend on how its packets meet the two kernels."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,prec,ipeel", [
    ("tiny", hc3d.PREC_MIXED, 0), ("tiny3d", hc3d.PREC_MIXED, 1), ("tiny_acc", hc3d.PREC_MIXED, 1),
    ("tiny_sg", hc3d.PREC_MIXED, 0), ("tiny3d", hc3d.PREC_FP64, 0), ("tiny_sg", hc3d.PREC_FP64, 1)])
def test_batches_of_any_size_sum_to_the_whole(tmp_path, built, name, prec, ipeel):
    """Shards of 1, 31, 33, 129 and the remaining packets -- one lane, a warp
    less one, a warp and one, a block and one, more packets than warps --
    add up to one run of all of them, every integer."""
    m = make_model(tmp_path, name, MAXINT=3000)
    n = 4000
    ctx = hc3d.Context(prec).load(m)
    it = 1 if m.sg else 3

    def run(off, k):
        p = m.run_params(np_total=n, np=k, iter=it, ipeel=ipeel, packet_offset=off)
        ctx.zero()
        ctx.run(p)
        return ctx.tallies(p)

    whole = run(0, n)
    total, off = None, 0
    for k in (1, 31, 33, 129, n - 194):
        t = run(off, k)
        off += k
        assert t["path_scale"] == whole["path_scale"]
        if total is None:
            total = {q: np.array(v) for q, v in t.items() if isinstance(v, np.ndarray)}
        else:
            for q in total:
                total[q] = total[q] + t[q]
    assert whole["counters"][hc3d.CNT["events"]] > n
    for q, v in total.items():
        np.testing.assert_array_equal(v, whole[q], err_msg=q)
    ctx.close()


@pytest.mark.parametrize("ipeel", [0, 1])
def test_interaction_cap_in_the_tail(tmp_path, built, ipeel):
    """A packet is killed at the cap on its interactions, wherever it is run."""
    m = make_model(tmp_path, "tiny_acc")
    ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
    n = 3000
    got = {}
    for cap in (1, 7, 200):
        p = m.run_params(np=n, iter=3, ipeel=ipeel, max_interactions=cap)
        ctx.zero()
        ctx.run(p)
        c = ctx.tallies(p)["counters"]
        assert c[hc3d.CNT["escaped"]] + c[hc3d.CNT["aflux"]] + c[hc3d.CNT["abflux"]] + c[hc3d.CNT["stuck"]] == n
        assert c[hc3d.CNT["events"]] <= cap * n
        got[cap] = c[hc3d.CNT["abflux"]]
    assert got[1] > got[7] > got[200] > 0
    ctx.close()
