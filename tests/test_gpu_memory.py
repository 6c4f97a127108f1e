"""Device memory that a loaded model holds, from the allocator's own count."""
from __future__ import annotations

import ctypes as C

import pytest

from hochunk3d_gb300 import hc3d
from tests.helpers import make_model

pytestmark = pytest.mark.gpu


def _used():
    """Bytes in use of the device's default pool (cudaMemPoolAttrUsedMemCurrent)."""
    import torch

    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.%s" % torch.version.cuda.split(".")[0])
    pool, n = C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(n)) == 0
    return n.value


def test_rows_of_the_mixed_form_are_not_kept_in_fp64(tmp_path, built):
    """The rows of the Lucy CDF (8 bytes per cell and species slot), which only
    the mixed form reads."""
    m = make_model(tmp_path, "plain")
    held = {}
    for prec in (hc3d.PREC_MIXED, hc3d.PREC_FP64):
        ctx = hc3d.Context(prec)
        before = _used()
        ctx.load(m)
        held[prec] = _used() - before
        ctx.close()
    rows = 4 * 8 * m.info.ncells
    assert held[hc3d.PREC_FP64] <= held[hc3d.PREC_MIXED] - rows, held


def test_tables_are_kept_once(tmp_path, built):
    """Of the Lucy CDF: the FP64 tables and, of the same size, the pairs of FP32
    rows that the mixed form draws from; 300 bytes a cell and 8 MB hold the rest."""
    m = make_model(tmp_path, "plain")
    ctx = hc3d.Context(hc3d.PREC_MIXED)
    before = _used()
    ctx.load(m)
    held = _used() - before
    ctx.close()
    assert held <= 2 * 4 * 8 * m.nT * m.nnu + 300 * m.info.ncells + (8 << 20), held


@pytest.mark.parametrize("name,over", [("tiny", {}), ("tiny_sg", {}), ("plain", {}), ("plain", {"NPG": 17})])
def test_footprint_covers_what_a_model_holds(tmp_path, built, name, over):
    """The server's admission size is at least the loaded model and the peeled
    iteration's SED and image tallies."""
    m = make_model(tmp_path, name, **over)
    ctx = hc3d.Context(hc3d.PREC_MIXED)
    before = _used()
    ctx.load(m)
    held = _used() - before
    p = m.run_params(np=100, iter=1, ipeel=1)
    ctx.zero()
    ctx.run(p)
    t = ctx.tallies(p, grid=False)
    ctx.close()
    tallies = sum(t[k].nbytes for k in t if k.startswith(("image", "s", "t", "num")) and hasattr(t[k], "nbytes"))
    assert int(hc3d.lib().hc3d_model_footprint(m._h)) >= held + tallies, (held, tallies)
