"""vpmg_dirichlet_static where its passes are products on the tensor cores:
along x only, along y only, along both (even and odd N), the line length at
which they begin, a box inside the node array, and a call with FFT passes
between two with products (all share the static array).

The products round the line's values and the sines to 55 bits of the line's
largest, the FFT passes to 53 bits a stage: the tolerance is that of the other
Dirichlet parity tests."""
import ctypes as C

import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-12

# (nz, ny, nx) of the box, its offset in the array, spacings, zero_bc
CASES = [((40, 31, 105), (0, 0, 0), (0.05, 0.07, 0.06), 0),
         ((36, 121, 33), (0, 0, 0), (0.05, 0.04, 0.06), 1),
         ((13, 17, 19), (1, 2, 3), (0.1, 0.2, 0.15), 0),
         ((14, 136, 101), (2, 1, 3), (0.03, 0.02, 0.04), 0),
         ((14, 136, 101), (1, 1, 1), (0.03, 0.02, 0.04), 1),
         ((5, 409, 391), (0, 0, 0), (0.01, 0.3, 0.2), 0)]


def test_products_match_oracle(gpulib, oracle):
    torch = pytest.importorskip("torch")
    L = gpulib.load_library()
    f = L.vpmg_dirichlet_static
    f.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_int), C.POINTER(C.c_int), C.POINTER(C.c_double), C.c_int,
                  C.c_void_p]
    f.restype = C.c_int
    rng = np.random.default_rng(5)
    for k, (shape, off, d, zero_bc) in enumerate(CASES):
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
        assert rel_l2(got[at], ref) <= TOL, (k, rel_l2(got[at], ref))
        got[at] = sol[at]  # nothing outside the box changed
        assert np.array_equal(got, sol), k
