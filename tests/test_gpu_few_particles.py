"""Mesh-to-particle below and above the number of particles where a particle
takes four lanes (77824): the same particles alone and inside a larger set.  The
sums run in another order: a particle's 64 products differ by the rounding of
64 additions, 64 x 2^-53 of the largest, 1e-14 of the fields' scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("few", [1, 3, 500, 77823])
def test_few_particles_take_the_same_values(gpulib, few):
    V = gpulib
    if V.arith != "fp64":
        pytest.skip("FP64 kernel")
    rng = np.random.default_rng(few)
    n = 77824 + 200
    xp = rng.uniform(0.45, 1.15, (n, 3))
    qp = np.concatenate([rng.standard_normal((n, 3)), np.full((n, 1), 1e-3)], axis=1)
    qp[few:, :3] = 0.0  # the others are probes: both sets deposit the same vorticity
    d = (0.05, 0.05, 0.05)
    out = []
    for m in (few, n):
        with V.VPM(V.VPMConfig.make(dpm=d, box=(0.0, 0.0, 0.0, 1.6, 1.6, 1.6))) as h:
            x, q = xp[:m].copy(), qp[:m].copy()
            h.vpm(x, q, None, None, m, WhatToDo=0, NTIME=0)
            up, gp = np.zeros((m, 3)), np.zeros((m, 3))
            h.vpm(x, q, up, gp, m, WhatToDo=2, NTIME=1)
            out.append((up[:few], gp[:few]))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-12 * max(np.abs(b).max(), 1e-300)
