"""Which DST passes go as products on the tensor cores (dst_mma_wanted in
csrc/dst_mma.cu), read through vpmg_dst_tiles, and their results on both sides
of the rule's lines.

Tolerance 1e-12, the Dirichlet bar of the parity tests (the reasoning is in
test_gpu_dst_products.py).
"""
import ctypes as C

import numpy as np
import pytest

from helpers import rel_l2
from test_gpu_dst_products import _reference, _solve

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


@pytest.mark.parametrize("cells,ncoarse,block,inner", [
    # lines of the padded block (cells + 2 ncoarse) and of the inner box, three components, tiles of 64
    ((96, 32, 32), 4, False, False),     # block: N = 104, 39 x 39 lines, 72 tiles
    ((96, 32, 40), 4, True, False),      # 39 x 47 lines, 86 tiles
    ((135, 24, 24), 3, False, False),    # odd inner lines: N = 135, 23 x 23, 25 tiles; block N = 141, 29 x 29, 40 tiles
    ((135, 36, 36), 3, True, True),      # 41 x 41 lines, 79 tiles; 35 x 35, 58 tiles
])
def test_few_lines_stay_with_the_fft(gpulib, cells, ncoarse, block, inner):
    if gpulib.arith != "fp64":
        pytest.skip("the products are FP64's")
    t = _tiles(gpulib, cells, ncoarse)
    assert (t["block_x"] == 0) == block and (t["inner_x"] == 0) == inner, t


# N and lines that take products: the tiles' and pieces' edges of test_gpu_dst_products.py with more planes
@pytest.mark.parametrize("shape", [
    (23, 102, 101),   # N = 100 along x (100 x 21 lines, 99 tiles), 101 along y
    (18, 130, 259),   # 129 odd outputs along x (96 tiles): a second tile of one row; N = 129 along y (193)
    (20, 114, 130),   # N = 129 and 113, odd
    (12, 260, 417),   # N = 416: the longest lines, pieces in two halves (122 tiles); 259 along y (195)
    (13, 418, 300),   # N = 417 along y: the last length as products (154 tiles, two rounds); 299 along x (215)
    (40, 65, 121),    # 63 x 38 lines: 113 tiles along x, FFT along y
])
def test_products_on_enough_lines(gpulib, shape):
    rng = np.random.default_rng(3)
    rhs = [rng.standard_normal(shape) for _ in range(3)]
    # values over twelve decades within and across lines, and planes without any
    rhs[1] *= 10.0 ** rng.uniform(-12, 0, (shape[0], shape[1], 1))
    rhs[2][:, :, : shape[2] // 2] = 0.0
    rhs[2][: shape[0] // 2] = 0.0
    sol = [rng.standard_normal(shape), np.zeros(shape), np.zeros(shape)]
    out = _solve(gpulib, rhs, sol)
    for c in range(3):
        assert rel_l2(out[c], _reference(rhs[c], sol[c])) <= 1e-12, c


def test_static_products_match_oracle(gpulib, oracle):
    """The allocation-free solve where its passes are products: along x alone, along
    y alone, along both (given and zero boundary values, a box inside the array),
    two pieces, and a call with FFT passes between."""
    torch = pytest.importorskip("torch")
    f = gpulib.load_library().vpmg_dirichlet_static
    f.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_int), C.POINTER(C.c_int), C.POINTER(C.c_double), C.c_int,
                  C.c_void_p]
    rng = np.random.default_rng(5)
    # (nz, ny, nx) of the box, its offset in the array, zero_bc; tiles of one component
    cases = [((92, 82, 105), (0, 0, 0), 0),   # x: N = 104, 113 tiles
             ((92, 121, 82), (0, 0, 0), 1),   # y: N = 120, 113 tiles
             ((13, 17, 19), (1, 2, 3), 0),
             ((82, 136, 101), (2, 1, 3), 0),  # x: N = 100, 168 tiles in two rounds (FFT); y: N = 135, 124
             ((112, 136, 121), (1, 1, 1), 1),  # both: 231 and 205 tiles
             ((30, 256, 273), (0, 0, 0), 0)]  # x: N = 272 in two pieces, 112 tiles; y: N = 255, 119
    for k, (shape, off, zero_bc) in enumerate(cases):
        d = (0.05, 0.07, 0.06)
        full = tuple(n + 2 * o for n, o in zip(shape, off))
        rhs, sol = rng.standard_normal(full), rng.standard_normal(full)
        at = tuple(slice(o, o + n) for n, o in zip(shape, off))
        a, b = torch.from_numpy(rhs).cuda(), torch.from_numpy(sol).cuda()
        lo, hi = off[::-1], [o + n - 1 for n, o in zip(shape, off)][::-1]
        rc = f(a.data_ptr(), b.data_ptr(), (C.c_int * 3)(*full[::-1]), (C.c_int * 6)(*lo, *hi), (C.c_double * 3)(*d),
               zero_bc, None)
        assert rc == 0, (k, rc)
        torch.cuda.synchronize()
        got = b.cpu().numpy()
        ref = np.ascontiguousarray(sol[at])
        oracle.dirichlet(np.ascontiguousarray(rhs[at]), ref, d, zero_bc=bool(zero_bc))
        assert rel_l2(got[at], ref) <= 1e-12, (k, rel_l2(got[at], ref))
        got[at] = sol[at]  # nothing outside the box changed
        assert np.array_equal(got, sol), k
