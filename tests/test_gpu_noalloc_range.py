"""hc3d_lucy_update_noalloc on the edges of what its buffers may hold, against
the fixed point of its equation in numpy: T = (na L / (4 sigma N kappa_V
kappa_P(T0)))^(1/4) / (11605 (rho V)^(1/4)), clamped to [0.1, 1600] K."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from hochunk3d_gb300 import hc3d

pytestmark = pytest.mark.gpu
LO, HI = 0.1 / 11605.0, 1600.0 / 11605.0


def _solve(tally, mass, t0, kp0=0.7):
    """Cells in a row (one more wall than cells along each axis); a gray
    species, kappa_P = kp0 everywhere, so that one step is the solution."""
    import torch

    n = len(tally)
    shape = (1, 2, 2, n + 1)
    dev = torch.device("cuda", 0)
    nT, ltot, npk, kv, scale = 50, 3.0e33, 1000000, 150.0, 2.0 ** 20
    lT = np.log(np.logspace(np.log10(LO), np.log10(HI), nT))

    def field(v, dtype):
        a = np.zeros(shape, dtype)
        a[0, 0, 0, :n] = v
        return a

    host = {"dtauabs": field(tally, np.int64), "densarr": field(1e-18, float), "massarr": field(mass, float),
            "tdust_in": field(t0, float), "lTint": lT, "kappap": np.full(nT, kp0)}
    keep = {q: torch.from_numpy(v).to(dev) for q, v in host.items()}
    out = torch.zeros(shape, dtype=torch.float64, device=dev)
    b = hc3d.LucyBuffers()
    b.device, b.stream = 0, torch.cuda.current_stream(dev).cuda_stream
    b.ndg, b.npg, b.ntg, b.nrg = shape
    for q, v in keep.items():
        setattr(b, q, v.data_ptr())
    b.tdust_out = out.data_ptr()
    b.path_scale, b.nT, b.ltot, b.np = scale, nT, ltot, npk
    b.kappav[0] = kv
    rel, conv = C.c_double(), C.c_int()
    assert hc3d.lib().hc3d_lucy_update_noalloc(C.byref(b), C.byref(rel), C.byref(conv)) == 0
    with np.errstate(all="ignore"):
        root = np.power(np.asarray(tally, float) / scale * ltot / (4.0 * 5.6704e-5 * npk * kv * kp0), 0.25) / 11605.0
        want = np.where(np.asarray(mass) > 0.0, root / mass, LO)
    return out.cpu().numpy()[0, 0, 0, :n], np.clip(want, LO, HI), rel.value


def test_negative_starting_temperature(built):
    """The solution does not depend on the start; one below zero lies below the
    table of opacities, as any start under 0.1 K does."""
    t0 = np.array([-1.0, -1e-300, -0.05, -1e300, 0.01])
    got, want, rel = _solve(np.full(5, 1 << 40), np.full(5, 1.0e6), t0)
    assert LO < want[0] < HI
    np.testing.assert_allclose(got, want, rtol=1e-12)  # the iterates agree to a few ulp
    assert np.isfinite(rel)


def test_masses_of_any_size(built):
    """A cell that absorbed nothing is at the floor and one that absorbed is
    where its mass puts it, however small or large the mass."""
    mass = np.array([1e-300, 1e-90, 1e-82, 1e-3, 1e5, 1e73, 1e90, 1e300, 5e-324])
    for tally in (0, 1 << 40):
        got, want, _ = _solve(np.full(len(mass), tally), mass, np.full(len(mass), 0.01))
        np.testing.assert_allclose(got, want, rtol=1e-12, err_msg=str(tally))


def _fixed_point(f, na, mass, t0, lT, kp, c):
    """The iteration in the floating-point type f of its operands."""
    na, mass, t0, lT, kp, c = (np.asarray(v, dtype=f) for v in (na, mass, t0, lT, kp, c))
    n = len(lT)
    lo, hi, eps = f(0.1) / f(11605), f(1600) / f(11605), f(1e-5)
    td, told = t0.copy(), f(0.5) * t0
    busy = np.ones(len(t0), bool)
    while busy.any():
        lt = np.log(td)
        k = ((n - 1) * (lt - lT[0]) / (lT[-1] - lT[0])).astype(int) + 1
        i = np.clip(k, 1, n - 1)
        w = (lt - lT[i - 1]) / (lT[i] - lT[i - 1])
        kap = np.where(k < 1, kp[0], np.where(k > n - 1, kp[-1], (1 - w) * kp[i - 1] + w * kp[i]))
        new = np.clip(np.power(na * c / kap, f(0.25)) / f(11605) / mass, lo, hi)
        told = np.where(busy, td, told)
        td = np.where(busy, new, td)
        busy &= np.abs(td - told) > eps * td
    return td


def test_error_against_extended_precision(tmp_path, built):
    """The solve's logarithm and fourth root are no further from the exact
    iterates than those of plain FP64: the root mean square of the relative
    error against the same iteration in extended precision is at most that of
    numpy's FP64 iteration (log and power of the C library)."""
    import torch

    from tests.helpers import make_model

    assert np.finfo(np.longdouble).eps < 1e-18
    m = make_model(tmp_path, "tiny", warm=False)
    rng = np.random.default_rng(11)
    n, npk, ltot, kv = 40000, 100000000, float(m.info.ltot), float(m.kappav[0])
    lT, kp = np.ascontiguousarray(m.lTint), np.ascontiguousarray(np.ravel(m.kappap)[: m.nT])
    t = np.clip(1500.0 * 150.0 ** -rng.random(n) * 10.0 ** rng.uniform(-0.3, 0.1, n), 10.0, 1500.0) / 11605.0
    mass = (10.0 ** rng.uniform(-22, -12, n) * 10.0 ** rng.uniform(36, 40, n)) ** 0.25
    c = np.longdouble(ltot) / (np.longdouble(4.0) * np.longdouble(5.6704e-5) * npk * np.longdouble(kv))
    scale = 2.0 ** 21
    tally = np.clip(np.round((t * 11605.0 * mass) ** 4 * np.interp(np.log(t), lT, kp) / float(c) * scale), 1.0, 9e15)
    tally = tally.astype(np.int64)
    t0 = np.clip(t * rng.uniform(0.7, 1.3, n), LO, HI)
    args = (tally / scale, mass, t0, lT, kp)
    exact = _fixed_point(np.longdouble, *args, c)
    plain = _fixed_point(np.float64, *args, ltot / (4.0 * 5.6704e-5 * npk * kv))

    shape = (1, 2, 2, n + 1)
    dev = torch.device("cuda", 0)

    def field(v, dtype=np.float64):
        a = np.zeros(shape, dtype)
        a[0, 0, 0, :n] = v
        return torch.from_numpy(a).to(dev)

    keep = {"dtauabs": field(tally, np.int64), "densarr": field(1e-18), "massarr": field(mass), "tdust_in": field(t0),
            "lTint": torch.from_numpy(lT).to(dev), "kappap": torch.from_numpy(kp).to(dev)}
    out = torch.zeros(shape, dtype=torch.float64, device=dev)
    b = hc3d.LucyBuffers()
    b.device, b.stream = 0, torch.cuda.current_stream(dev).cuda_stream
    b.ndg, b.npg, b.ntg, b.nrg = shape
    for q, v in keep.items():
        setattr(b, q, v.data_ptr())
    b.tdust_out = out.data_ptr()
    b.path_scale, b.nT, b.ltot, b.np = scale, m.nT, ltot, npk
    b.kappav[0] = kv
    rel, conv = C.c_double(), C.c_int()
    assert hc3d.lib().hc3d_lucy_update_noalloc(C.byref(b), C.byref(rel), C.byref(conv)) == 0
    got = out.cpu().numpy()[0, 0, 0, :n]

    def rms(x):
        return float(np.sqrt(np.mean(((x - exact) / exact).astype(np.float64) ** 2)))

    assert rms(got) <= rms(plain), (rms(got), rms(plain))
