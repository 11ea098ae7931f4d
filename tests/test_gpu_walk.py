"""pmesh's boundary values by one walk of the quadtree, against the oracle.

The walk's coarsest cells are cut into segments by the number of targets, so
the sizes run from one segment of a tiny mesh over ragged faces (dummy cells on
one side or both) to several segments.
Tolerance: relative L2 <= 1e-10 (fields), as for the solves.
"""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


# (nz, ny, nx), levmax, tree
CASES = [((9, 9, 9), 1, 1), ((10, 9, 11), 2, 1), ((17, 20, 23), 2, 1), ((35, 33, 38), 3, 1), ((33, 41, 49), 3, 1),
         ((12, 9, 14), 0, 0), ((12, 15, 14), 0, 1)]


@pytest.mark.parametrize("ibctyp", [2, 3])
@pytest.mark.parametrize("shape,levmax,tree", CASES)
def test_one_walk_matches_oracle(gpulib, oracle, shape, levmax, tree, ibctyp):
    V = gpulib
    rng = np.random.default_rng(sum(shape) + levmax)
    d = (0.06, 0.05, 0.07)
    nz, ny, nx = shape
    xb = (-0.3, 0.1, 0.0, -0.3 + (nx - 1) * d[0], 0.1 + (ny - 1) * d[1], (nz - 1) * d[2])
    rhs = [rng.standard_normal(shape) for _ in range(3)]
    ref = [np.zeros(shape) for _ in range(3)]
    oracle.pmesh(ref, rhs, xb, d, iynbc=1, itree=tree, levmax=levmax, ibctyp=ibctyp)
    cfg = V.VPMConfig.make(dpm=d, box=(0, 0, 0, d[0] * 8, d[1] * 8, d[2] * 8), ibctyp=ibctyp)
    with V.VPM(cfg) as h:
        out = [np.zeros(shape) for _ in range(3)]
        h.pmesh(out, rhs, xb, d, iynbc=1, itree=tree, levmax=levmax)
    for c in range(3):
        assert rel_l2(out[c], ref[c]) <= 1e-10, c
