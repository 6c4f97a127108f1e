"""The memory that an unpeeled run keeps for the packets it leaves to the
warp-per-packet kernel: no more than there are such packets."""
from __future__ import annotations

import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


def test_a_large_launch_of_few_packets(tmp_path, built):
    """100000 blocks of 128 threads are accepted for 3000 packets; the room is
    the packets' (3000 places of at most 512 bytes), not the threads'."""
    import torch

    m = make_model(tmp_path, "tiny", MAXINT=500)
    p = m.run_params(np=3000, iter=3, ipeel=0)
    want = None
    free = []
    for blocks in (0, 100000):
        ctx = hc3d.Context(hc3d.PREC_MIXED, grid_blocks=blocks).load(m)
        ctx.zero()
        before = torch.cuda.mem_get_info(0)[0]
        ctx.run(p)
        free.append(before - torch.cuda.mem_get_info(0)[0])
        t = ctx.tallies(p)
        ctx.close()
        if want is None:
            want = t
        assert (t["dtauabs"] == want["dtauabs"]).all() and (t["counters"] == want["counters"]).all()
    # the pool of stream-ordered memory grows in pieces of tens of megabytes
    assert free[1] < free[0] + (256 << 20), free
