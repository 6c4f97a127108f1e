"""Models whose species have dust files of their own: more than one table, in
shared memory, in shared memory for one kernel only, and in global memory."""
from __future__ import annotations

import numpy as np
import pytest

from hochunk3d_gb300 import configs, hc3d
from tests.helpers import splitmix_uniforms, trace_key, warm_tdust

pytestmark = pytest.mark.gpu


def _model(tmp_path, rows):
    """The tiny model, its envelope and cavity with grains of `rows`
    wavelengths: bluer, brighter and more forward scattering."""
    d = tmp_path
    configs.write_fixtures(d)
    lam = 10.0 ** np.linspace(-2.0, 4.0, rows)
    x = np.clip((np.log10(lam) + 1.0) / 2.0, 0.0, 1.0)
    kap = 140.0 * (0.55 / np.maximum(lam, 0.1)) ** 1.3
    with open(d / "other_dust.par", "w") as f:
        for l, k, a, g in zip(lam, kap, 0.7 * (1.0 - x), 0.75 * (1.0 - x)):
            f.write(f" {l:.6e} {k * 1e-22:.6e} {a * k * 1e-22:.6e} {k:.6e} {g:.6e} {0.4:.6e} {0.0:.6e}\n")
    other = {f"DUSTNAME({k})": "other_dust.par" for k in (3, 4, 7, 8)}
    m = hc3d.Model(configs.write_par(d, "tiny", MAXINT=2000, **other))
    m.set_tdust(warm_tdust(m))
    return m


# the 241 rows of the usual file and: as many, enough to leave the tail kernel's shared memory, all shared memory
@pytest.mark.parametrize("rows", [241, 900, 1000])
def test_two_dust_files(tmp_path, built, rows):
    import oracle.oracle as O

    m = _model(tmp_path, rows)
    nu = 6000
    U = splitmix_uniforms(24, nu, seed=41)
    pt = m.run_params(np=24, iter=3, ipeel=0)
    traces = {}
    for prec in (hc3d.PREC_FP64, hc3d.PREC_MIXED):
        ctx = hc3d.Context(prec).load(m)
        traces[prec] = [trace_key(t) for t in ctx.trace(pt, U, max_rec=2048)]
        ctx.close()
    same = 0
    for k in range(24):
        want, ended, _ = O.trace(m, pt, k, U[k], max_rec=2048)
        if not ended:  # the draws sufficed
            np.testing.assert_array_equal(traces[hc3d.PREC_FP64][k], trace_key(want), err_msg=str(k))
        same += int(np.array_equal(traces[hc3d.PREC_MIXED][k], traces[hc3d.PREC_FP64][k]))
    assert same >= 18  # as with one table
    n = 3000
    p = m.run_params(np=n, iter=3, ipeel=0)
    for prec in (hc3d.PREC_FP64, hc3d.PREC_MIXED):
        got = []
        for blocks in (1, 0):  # nearly all events in k_wave, in k_tail
            ctx = hc3d.Context(prec, grid_blocks=blocks).load(m)
            ctx.zero()
            ctx.run(p)
            got.append(ctx.tallies(p))
            ctx.close()
        for key, v in got[0].items():
            if isinstance(v, np.ndarray):
                np.testing.assert_array_equal(v, got[1][key], err_msg=key)
        if prec == hc3d.PREC_FP64:
            r = O.run(m, p)
            for k in (0, 4, 5, 6, 9, 12, 13, 14):  # last-ulp branch flips of the device transcendentals
                assert abs(int(got[0]["counters"][k]) - int(r["counters"][k])) <= 2 + 0.002 * abs(int(r["counters"][k])), k
