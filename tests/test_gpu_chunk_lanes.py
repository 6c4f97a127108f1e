"""A small chunk of a peeled iteration after one that filled the pool: its
packets start in whatever lanes are free, beside the histories carried over."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regen", [1, 4, 16])
def test_small_chunk_after_a_full_one(tmp_path, built, regen):
    """100 packets after 600000: started within a few waves of a dozen events,
    not after the carried histories of up to 3000 events have ended, and the
    tallies are those of one run of all."""
    m = make_model(tmp_path, "plain", MAXINT=3000, MASSD=0.1, NPEEL=1, THETE="45.0", PHIE="0.0", NXIMG=31)
    n, first = 600100, 600000
    ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
    ctx.set_wave_options(queue_records=1 << 20, regen=regen)
    whole = m.run_params(np=n, iter=3, ipeel=1)
    ctx.zero()
    ctx.run(whole)
    want = ctx.tallies(whole)
    ctx.zero()
    ctx.run_chunk(m.run_params(np_total=n, np=first, iter=3, ipeel=1), n, final=False)
    carried = ctx.wave_log()[-1, 2]
    assert carried > 30000  # packets in flight, in most lanes of the pool
    ctx.run_chunk(m.run_params(np_total=n, np=n - first, iter=3, ipeel=1, packet_offset=first), n, final=False)
    waves = len(ctx.wave_log())
    ctx.run_chunk(m.run_params(np_total=n, np=0, iter=3, ipeel=1, packet_offset=n), n, final=True)
    got = ctx.tallies(whole)
    ctx.close()
    for key in ("si", "nums", "ti", "numt", "image_i", "nabs", "dtauabs", "jmean", "killed", "counters"):
        np.testing.assert_array_equal(got[key], want[key], err_msg=key)
    assert waves <= 4, waves
