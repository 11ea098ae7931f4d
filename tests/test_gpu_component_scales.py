"""Components of very different size through one vector-potential solve: they share
the boundary operator's complex transforms, not each other's rounding.

A component times a power of two gives its solution times that power, to the last
bit: every step of the solve is linear in it, and scaled to the component itself.
A component of zeros stays zero, one with a value that is not finite keeps to
itself; the others agree with the plain solve to rounding, 1e-13 (float-float
1e-12).
"""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def solved(gpulib):
    cells, h = (48, 0.05) if gpulib.arith == "fp64" else (96, 0.05)  # both go by FFT and tables
    cfg = gpulib.VPMConfig.make(dpm=(h,) * 3, box=(0.0, 0.0, 0.0) + (cells * h,) * 3)
    H = gpulib.VPM(cfg)
    H.define_sizes(np.full((1, 3), 0.5 * cells * h))
    assert H.farfield_stats()["on"]
    r = np.random.default_rng(2).standard_normal((3,) + (cells + 1,) * 3)
    yield gpulib, H, r, H.apply_poisson(r)
    H.close()


@pytest.mark.parametrize("powers", [(0, -30, 0), (-30, 0, 0), (0, 0, -40), (20, -20, 3), (-70, 0, 70)])
def test_powers_of_two(solved, powers):
    V, H, r, unit = solved
    if V.arith != "fp64" and max(map(abs, powers)) > 50:
        pytest.skip("outside the floats' range of products")
    s = np.exp2(np.array(powers, dtype=np.float64)).reshape(3, 1, 1, 1)
    psi = H.apply_poisson(r * s)
    for c in range(3):
        assert np.array_equal(psi[c], unit[c] * s[c]), (c, rel_l2(psi[c], unit[c] * s[c]))


@pytest.mark.parametrize("c", [0, 1, 2])
def test_a_component_of_zeros(solved, c):
    V, H, r, unit = solved
    q = r.copy()
    q[c] = 0.0
    psi = H.apply_poisson(q)
    assert not psi[c].any()
    for k in {0, 1, 2} - {c}:
        assert rel_l2(psi[k], unit[k]) <= (1e-13 if V.arith == "fp64" else 1e-12)


@pytest.mark.parametrize("c", [0, 1, 2])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_component_that_is_not_finite(solved, c, bad):
    V, H, r, unit = solved
    if V.arith != "fp64":
        pytest.skip("float-float has no infinities or NaN")
    q = r.copy()
    q[c, 20, 21, 22] = bad
    psi = H.apply_poisson(q)
    assert not np.isfinite(psi[c][1:-1, 1:-1, 1:-1]).any()
    for k in {0, 1, 2} - {c}:
        assert rel_l2(psi[k], unit[k]) <= 1e-13
