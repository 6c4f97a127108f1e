"""The scattering of the mixed form rounds as its source says.

A packet's history may pass from one thread to a warp anywhere, so both have to
scatter it to the same bits.  They do where no product is left for the compiler
to fuse with a sum, or not, as it likes: ``tests/scatter.cu`` is compiled with
contraction on and off, and a thread and a warp leave the same packet in both."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from hochunk3d_gb300 import build as B

pytestmark = pytest.mark.gpu
EVENT = np.dtype([(k, "f4") for k in ("cost", "sint", "phi", "cosp", "sinp", "sip", "sqp", "sup", "svp", "g", "pl")]
                 + [("kapd", "f4", 4), ("rho", "f4", 4), ("u", "f4"), ("pid", "u4")])
LEFT = np.dtype([(k, "f4") for k in ("cost", "sint", "phi", "cosp", "sinp", "sip", "sqp", "sup", "svp", "mu", "smu",
                                     "rprob")] + [("species", "i4"), ("draws", "i4")])


def _events(n, glo, ghi):
    rng = np.random.default_rng(11)
    e = np.zeros(n, EVENT)
    e["cost"] = rng.uniform(-1.0, 1.0, n)
    e["cost"][:4] = (1.0, -1.0, 0.0, 1.0 - 2.0 ** -24)
    e["sint"] = np.sqrt(1.0 - e["cost"].astype(float) ** 2)
    phi = rng.uniform(0.0, 2.0 * np.pi, n)
    e["phi"], e["cosp"], e["sinp"] = phi, np.cos(phi), np.sin(phi)
    e["sip"] = rng.uniform(0.5, 2.0, n)
    for k in ("sqp", "sup", "svp"):
        e[k] = rng.uniform(-0.5, 0.5, n) * e["sip"]
    e["g"], e["pl"] = rng.uniform(glo, ghi, n), rng.uniform(0.0, 1.0, n)
    e["kapd"] = 10.0 ** rng.uniform(-3, 2, (n, 4))
    e["rho"] = 10.0 ** rng.uniform(-3, 2, (n, 4)) * (rng.uniform(size=(n, 4)) < 0.7)
    # selection draws within a few units of the last place of a species' boundary
    k = e["kapd"].astype(float) * e["rho"]
    cum = np.cumsum(k, 1) / np.where(k.sum(1) > 0.0, k.sum(1), 1.0)[:, None]
    e["u"] = np.clip(cum[np.arange(n), rng.integers(0, 4, n)] * (1.0 + rng.integers(-3, 4, n) * 2.0 ** -24), 1e-6, 1.0)
    e["pid"] = np.arange(n)
    return e


@pytest.fixture(scope="module")
def builds(tmp_path_factory):
    d = tmp_path_factory.mktemp("scatter")
    libs = []
    for k, flags in enumerate(([], ["--fmad=false"])):
        so = d / f"scatter{k}.so"
        subprocess.run([B._nvcc(), *B.ARCH, *B.NVCC_COMMON, *flags, "-shared", "-I", str(B.CSRC), "-I",
                        str(B.ROOT / "include"), "-o", str(so), str(B.ROOT / "tests" / "scatter.cu")], check=True,
                       capture_output=True)
        libs.append(C.CDLL(str(so)))
    return libs


@pytest.mark.parametrize("glo, ghi", [(-0.3, 0.3), (0.3, 0.95)])
def test_contraction_does_not_reach_the_scattering(builds, glo, ghi):
    import torch

    n = 100000
    e = _events(n, glo, ghi)
    d = torch.from_numpy(np.frombuffer(e.tobytes(), dtype=np.uint8).copy()).cuda()
    got = []
    for lib in builds:
        a, b = (torch.zeros(n * LEFT.itemsize, dtype=torch.uint8, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        assert lib.scatter(C.c_void_p(d.data_ptr()), n, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())) == 0
        got += [np.frombuffer(x.cpu().numpy().tobytes(), dtype=LEFT) for x in (a, b)]
    for k in LEFT.names:
        want = got[0][k].view("u4")
        differ = [int((g[k].view("u4") != want).sum()) for g in got[1:]]
        assert differ == [0, 0, 0], (k, differ)
