"""Which DST passes go as products on the tensor cores (dst_mma_wanted in
csrc/dst_mma.cu), read through vpmg_dst_tiles, and their results on both sides
of the rule's lines.

Tolerance 1e-12, the Dirichlet bar of the parity tests (the reasoning is in
test_gpu_dst_products.py).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tiles(V, cells, ncoarse=8):
    h = 0.02
    box = (0.0, 0.0, 0.0) + tuple(c * h for c in cells)
    with V.VPM(V.VPMConfig.make(dpm=(h,) * 3, box=box, ncoarse=ncoarse)) as H:
        H.define_sizes(np.array([[0.5 * c * h for c in cells]]))
        return H.dst_tiles()


def test_tiles_are_zero_where_passes_are_products(gpulib):
    """128^3: block lines of 144 intervals and inner lines of 128 go as products,
    the coarse grid's by FFT; 32^3 has no line long enough."""
    t = _tiles(gpulib, (128, 128, 128))
    fp64 = gpulib.arith == "fp64"
    for k in ("block_x", "block_y", "inner_x", "inner_y"):
        assert (t[k] == 0) if fp64 else (t[k] in (2, 4, 8)), (k, t)
    assert t["coarse_x"] in (2, 4, 8) and t["coarse_y"] in (2, 4, 8)
    assert all(v in (2, 4, 8) for v in _tiles(gpulib, (32, 32, 32)).values())
