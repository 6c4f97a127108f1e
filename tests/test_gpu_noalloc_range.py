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
