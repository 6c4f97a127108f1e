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


def test_temperature_solve_over_its_range(built):
    """hc3d_lucy_update_noalloc against the fixed point of the same equation in
    numpy (FP64, log and power of the C library): tallies of 1e-3 to 1e9
    absorbed-path units, starts far from the solution, empty cells, no tally,
    more opacity rows than the kernel keeps in shared memory.  The iterates
    agree to a few ulp, so the solutions do to 1e-12."""
    import ctypes as C

    import torch

    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(5)
    for nT in (7, 1000, 1500):
        lT = np.log(np.logspace(np.log10(0.1 / 11605.0), np.log10(1600.0 / 11605.0), nT))
        kp = np.exp(rng.normal(0.0, 0.3, nT).cumsum() * (0.02 if nT > 10 else 0.1) - 1.0)
        shape = (2, 5, 31, 41)  # (ndg, npg, ntg, nrg)
        na = 10.0 ** rng.uniform(-3, 9, shape)
        na[rng.random(shape) < 0.1] = 0.0
        scale = 2.0 ** 20
        tally = np.round(na * scale).astype(np.int64)
        na = tally / scale
        dens = np.where(rng.random(shape) < 0.2, 0.0, 1e-18)
        mass = 10.0 ** rng.uniform(3, 6, shape)
        mass[rng.random(shape) < 0.05] = 0.0
        t0 = 10.0 ** rng.uniform(np.log10(0.1), np.log10(1600.0), shape) / 11605.0
        ltot, npk, kv = 3.0e33, 1000000, 150.0
        lo, hi = 0.1 / 11605.0, 1600.0 / 11605.0
        td, told, busy = t0.copy(), 0.5 * t0, np.ones(shape, bool)
        for _ in range(1000):
            busy &= np.abs(td - told) > 1e-5 * td
            if not busy.any():
                break
            k = ((nT - 1) * (np.log(td) - lT[0]) / (lT[-1] - lT[0])).astype(int) + 1
            i = np.clip(k, 1, nT - 1)
            f = (np.log(td) - lT[i - 1]) / (lT[i] - lT[i - 1])
            kap = np.where(k < 1, kp[0], np.where(k > nT - 1, kp[-1], (1 - f) * kp[i - 1] + f * kp[i]))
            new = np.power(na * ltot / (4.0 * 5.6704e-5 * npk * kv * kap), 0.25) / 11605.0
            with np.errstate(divide="ignore", invalid="ignore"):
                new = np.clip(np.where(mass > 0.0, new / mass, lo), lo, hi)
            told = np.where(busy, td, told)
            td = np.where(busy, new, td)
        live = dens > 0.0
        live[:, -1] = live[:, :, -1] = live[:, :, :, -1] = False
        want = np.where(live, td, t0)
        keep = {"dtauabs": tally, "densarr": dens, "massarr": mass, "tdust_in": t0, "lTint": lT,
                "kappap": np.concatenate([kp, kp])}
        keep = {q: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for q, v in keep.items()}
        out = torch.zeros(shape, dtype=torch.float64, device=dev)
        b = hc3d.LucyBuffers()
        b.device, b.stream = 0, torch.cuda.current_stream(dev).cuda_stream
        b.ndg, b.npg, b.ntg, b.nrg = shape
        for q, v in keep.items():
            setattr(b, q, v.data_ptr())
        b.tdust_out = out.data_ptr()
        b.path_scale, b.nT, b.ltot, b.np = scale, nT, ltot, npk
        b.kappav[0] = b.kappav[1] = kv
        rel, conv = C.c_double(), C.c_int()
        assert hc3d.lib().hc3d_lucy_update_noalloc(C.byref(b), C.byref(rel), C.byref(conv)) == 0
        np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-12, err_msg=str(nT))
