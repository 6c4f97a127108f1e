"""The change of layout on the device, between the callers' (nrg,ntg,npg,ndg)
arrays and the cells between the walls, against the host's loops of
``hc3d_load_grid`` and ``hc3d_set_lucy_tally``: bytes are moved, so equal."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu

GRIDS = [("tiny", {}), ("tiny3d", {}), ("tiny_sg", {}), ("tiny", {"NRG": 33, "NTG": 17, "NPG": 2}),
         ("plain", {"NRG": 150, "NTG": 121, "NPG": 17})]


def _field(m, rng):
    td = np.asfortranarray(rng.uniform(10.0, 1500.0, m.shape4) / 11605.0)
    td[rng.uniform(size=m.shape4) < 0.1] = 0.0  # stands for the floor
    return td


@pytest.mark.parametrize("name,over", GRIDS)
def test_layouts_agree(tmp_path, built, name, over):
    m = make_model(tmp_path, name, MAXINT=200, **over)
    rng = np.random.default_rng(5)
    td = _field(m, rng)
    td[-1], td[:, -1], td[:, :, -1] = np.nan, -1.0, np.inf  # no cell lies beyond the last walls
    p = m.run_params(np=500, iter=1 if m.sg else 3, ipeel=0)
    ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
    ctx.set_tdust(td)
    clean = np.nan_to_num(td, nan=0.1 / 11605.0, posinf=0.1 / 11605.0)
    m.set_tdust(np.where(clean > 0.0, clean, 0.1 / 11605.0))
    other = hc3d.Context(hc3d.PREC_MIXED).load(m)
    out = []
    for c in (ctx, other):
        c.zero()
        c.run(p)
        t = c.tallies(p)
        t["td"], t["rel"], _ = c.lucy_update(m.info.ltot, 500)
        out.append(t)
    for q in out[0]:
        np.testing.assert_array_equal(out[0][q], out[1][q], err_msg=q)
    slots = [s - 1 for s in m.slot_species if s <= m.shape4[3]]
    cell = np.zeros(m.shape4, dtype=bool)
    cell[:-1, :-1, :-1] = True
    for q in ("nabs", "dtauabs"):
        assert not out[0][q][~cell].any()
    assert (out[0]["td"][~cell] == 0.1 / 11605.0).all()
    assert out[0]["jmean"].any() and out[0]["jmean"][cell[..., 0]].sum() == out[0]["jmean"].sum()
    # every place of the absorbed-path tally, with values of all 64 bits
    tally = np.asfortranarray(rng.integers(0, 1 << 62, m.shape4, dtype=np.int64))
    ctx.set_lucy_tally(tally)
    want = np.zeros_like(tally)
    for s in slots:
        want[:-1, :-1, :-1, s] = tally[:-1, :-1, :-1, s]
    np.testing.assert_array_equal(ctx.tallies(p)["dtauabs"], want)
    ctx.close()
    other.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -1e-30])
def test_a_refused_field_leaves_the_old_one(tmp_path, built, bad):
    m = make_model(tmp_path, "tiny3d", MAXINT=200)
    rng = np.random.default_rng(6)
    td = _field(m, rng)
    p = m.run_params(np=500, iter=3, ipeel=0)
    ctx = hc3d.Context(hc3d.PREC_MIXED).load(m)
    got = []
    for _ in range(2):
        ctx.set_tdust(td)
        if got:
            wrong = _field(m, rng)
            wrong[-2, -2, -2, 3] = bad
            with pytest.raises(hc3d.Hc3dError):
                ctx.set_tdust(wrong)
        ctx.zero()
        ctx.run(p)
        got.append(ctx.tallies(p))
        ctx.lucy_update(m.info.ltot, 500)
    for q in got[0]:
        np.testing.assert_array_equal(got[0][q], got[1][q], err_msg=q)
    ctx.close()
