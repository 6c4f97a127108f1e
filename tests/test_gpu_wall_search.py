"""The wall searches of the mixed form against each other, ray by ray.

A packet's history may pass from one thread (``next_wall_ray``) to a warp
(``next_wall_warp``) anywhere, so the two searches have to return the same
wall and the same distance, bit for bit, for every operand -- subnormal ones
included.  ``tests/wall_search.cu`` calls both on the same rays, and the
peel-off walk's roots of a cone."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from hochunk3d_gb300 import build as B

pytestmark = pytest.mark.gpu
RAY = np.dtype([(k, "f4") for k in ("x", "y", "z", "ux", "uy", "uz")] + [(k, "i4") for k in ("ir", "it", "ip", "own")])
CONE = np.dtype([(k, "f4") for k in ("c2", "hemi", "p2", "cz", "uz", "t")])
FOUND = np.dtype([("ok", "i4"), ("dt", "f4"), ("iface", "i4")])


@pytest.fixture(scope="module")
def searches(tmp_path_factory):
    so = tmp_path_factory.mktemp("walls") / "wall_search.so"
    subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_COMMON, "-shared", "-I", str(B.CSRC), "-I", str(B.ROOT / "include"),
                    "-o", str(so), str(B.ROOT / "tests" / "wall_search.cu")], check=True, capture_output=True)
    return C.CDLL(str(so))


def _dev(a):
    import torch

    return torch.from_numpy(np.frombuffer(a.tobytes(), dtype=np.uint8).copy()).cuda()


def _grid(scale):
    r = 1.0 + 99.0 * np.linspace(0.0, 1.0, 41) ** 2
    th = np.linspace(0.0, np.pi, 31)
    ph = np.linspace(0.0, 2.0 * np.pi, 9)
    tan2 = np.tan(th) ** 2
    tan2[[0, -1]] = 0.0          # the poles
    tan2[15] = -1.0              # the midplane
    hemi = np.where(np.cos(th) > 0.0, 1.0, -1.0)
    hemi[15] = -1.0
    r2 = (r * scale) ** 2
    w = np.concatenate([np.stack([r2[:-1], r2[1:]], 1), np.stack([tan2, hemi], 1),
                        np.stack([np.sin(ph), -np.cos(ph)], 1)]).astype(np.float32)
    return r * scale, th, ph, r2, w


def _rays(rng, n, scale, r, th, ph):
    q = np.zeros(n, RAY)
    q["ir"], q["it"], q["ip"] = rng.integers(1, 41, n), rng.integers(1, 31, n), rng.integers(1, 9, n)

    def inside(w, k):
        return w[k - 1] + (w[k] - w[k - 1]) * rng.uniform(1e-7, 1.0 - 1e-7, n)

    rr, tt, pp = inside(r, q["ir"]), inside(th, q["it"]), inside(ph, q["ip"])
    q["x"], q["y"], q["z"] = rr * np.sin(tt) * np.cos(pp), rr * np.sin(tt) * np.sin(pp), rr * np.cos(tt)
    mu, az = rng.uniform(-1.0, 1.0, n), rng.uniform(0.0, 2.0 * np.pi, n)
    q["ux"], q["uy"], q["uz"] = np.sqrt(1 - mu * mu) * np.cos(az), np.sqrt(1 - mu * mu) * np.sin(az), mu
    own = rng.integers(0, 7, n)  # on no wall, or on one of the six
    q["own"] = np.where(own == 0, 0, 1 << own)
    tiny = (rng.integers(-(1 << 22), 1 << 22, n).astype(np.float64) * 2.0 ** -149).astype(np.float32)
    k = rng.integers(0, 8, n)
    # beside the midplane and beside the planes phi = 0 and pi, a subnormal distance away
    q["z"] = np.where(k == 0, tiny, q["z"])
    q["it"] = np.where(k == 0, 15 + rng.integers(0, 2, n), q["it"])
    q["y"] = np.where(k == 1, tiny, q["y"])
    q["ip"] = np.where(k == 1, rng.choice([1, 4, 5, 8], n), q["ip"])
    # nearly along the axis, and nearly in the midplane
    q["ux"] = np.where(k == 2, tiny, q["ux"])
    q["uy"] = np.where(k == 2, 0.0, q["uy"])
    q["uz"] = np.where(k == 2, 1.0, np.where(k == 3, tiny, q["uz"]))
    return q


@pytest.mark.parametrize("fused", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -50, 2.0 ** -58, 2.0 ** 40])
def test_a_thread_and_a_warp_find_the_same_wall(searches, scale, fused):
    import torch

    r, th, ph, r2, w = _grid(scale)
    n = 100000
    q = _rays(np.random.default_rng(7), n, scale, r, th, ph)
    d_r2, d_w, d_q = _dev(r2), _dev(w), _dev(q)
    a, b = (torch.zeros(n * FOUND.itemsize, dtype=torch.uint8, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    assert searches.wall_search(len(r), len(th), len(ph), *(C.c_void_p(x.data_ptr()) for x in (d_r2, d_w, d_q)), n,
                                fused, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())) == 0
    one, many = (np.frombuffer(x.cpu().numpy().tobytes(), dtype=FOUND) for x in (a, b))
    assert one["ok"].mean() > 0.9
    differ = (one["ok"] != many["ok"]) | (one["dt"] != many["dt"]) | (one["iface"] != many["iface"])
    assert not differ.any(), (int(differ.sum()), q[differ][:3], one[differ][:3], many[differ][:3])


def test_cone_that_is_grazed_within_a_subnormal_discriminant(searches):
    """The discriminant C (cz^2 - a p^2) of rays that touch a cone next to the
    origin is subnormal; what the walk then takes for roots are roots: each
    satisfies |root - root in 64 bits| <= sqrt(2^-126) / |a|, the distance of
    the two roots where the discriminant leaves the normal range."""
    import torch

    rng = np.random.default_rng(3)
    n = 20000
    q = np.zeros(n, CONE)
    q["c2"], q["uz"], q["hemi"] = rng.uniform(0.3, 0.9, n), rng.uniform(-0.5, 0.5, n), rng.choice([-1.0, 1.0], n)
    q["cz"] = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-19.4, -18.5, n)
    a = q["c2"].astype(float) - q["uz"].astype(float) ** 2
    q["p2"] = q["cz"].astype(float) ** 2 / a * (1.0 - 10.0 ** rng.uniform(-6, -1, n))
    q["t"] = -1.0
    D = q["c2"].astype(float) * (q["cz"].astype(float) ** 2 - a * q["p2"].astype(float))
    sub = (a > 0.01) & (D > 0.0) & (D < 2.0 ** -127)
    assert sub.sum() > 1000
    d_q = _dev(q)
    out = torch.zeros(2 * n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert searches.cone_search(C.c_void_p(d_q.data_ptr()), n, C.c_void_p(out.data_ptr())) == 0
    roots = out.cpu().numpy().reshape(n, 2)[sub].astype(float)
    h = -(q["cz"].astype(float) * q["uz"].astype(float))[sub]
    mid = -h / a[sub]
    got = roots < 1e30
    off = np.abs(roots - mid[:, None])
    bound = 2.0 ** -63 / a[sub][:, None]
    assert (off[got] <= np.broadcast_to(bound, off.shape)[got]).all(), (off[got].max(), bound.max())
