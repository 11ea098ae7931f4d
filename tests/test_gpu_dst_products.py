"""Dirichlet solves where the DST passes go as matrix products (N >= 100
intervals along x or y, 1024 lines or more) and where the z sweep is short,
against scipy's DST-I and the same eigenvalues along all three axes.

Tolerance 1e-12, the Dirichlet bar of the parity tests: a pass rounds a
line's values and the sines to 2^-55 of the line's largest (a relative error
of 2^-54 sqrt(K) max / rms <= 2e-14 for K <= 208 folded values and
max / rms <= 20), four passes and the sweep stay below 1e-13.
"""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu
D = (0.05, 0.06, 0.04)


def _solve(V, rhs, sol):
    shape = rhs[0].shape
    with V.VPM(V.VPMConfig.make(dpm=D, box=(0, 0, 0, 0.4, 0.48, 0.32))) as h:
        out = [s.copy() for s in sol]
        h.pmesh(out, rhs, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), D, iynbc=0, NN_bl=(1, 1, 1) + shape[::-1])
    return out


def _reference(rhs, sol):
    from scipy.fft import dstn, idstn
    out = sol.copy()
    f = rhs[1:-1, 1:-1, 1:-1].copy()
    for ax, d in ((0, D[2]), (1, D[1]), (2, D[0])):
        for side, at in ((0, 0), (-1, -1)):
            face = sol[tuple(side if k == ax else slice(1, -1) for k in range(3))]
            f[tuple(at if k == ax else slice(None) for k in range(3))] -= face / d ** 2
    lam = 0.0
    for ax, d in ((0, D[2]), (1, D[1]), (2, D[0])):
        n = f.shape[ax]
        mu = 4.0 * np.sin(np.pi * np.arange(1, n + 1) / (2.0 * (n + 1))) ** 2 / d ** 2
        lam = lam - mu.reshape([-1 if k == ax else 1 for k in range(3)])
    out[1:-1, 1:-1, 1:-1] = idstn(dstn(f, type=1) / lam, type=1)
    return out


@pytest.mark.parametrize("shape", [
    (14, 102, 101),   # N = 100 (even) along x, 101 (odd) along y; lines not a multiple of the tile
    (11, 130, 259),   # 129 odd outputs along x: a second tile of one row; N = 129 along y
    (12, 114, 130),   # N = 129 along x (64 + 64 outputs), 113 along y
    (6, 260, 417),    # N = 416: the longest lines, pieces in two halves
    (6, 418, 300),    # N = 417 along y: the last length as products; 299 along x
    (6, 420, 300),    # N = 419: the FFT along y
])
def test_long_lines(gpulib, shape):
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


@pytest.mark.parametrize("nz", [3, 4, 5, 6, 7, 12, 13])
def test_short_sweeps(gpulib, nz):
    """1 to 11 planes: the two-ended elimination's middle, odd and even."""
    rng = np.random.default_rng(nz)
    shape = (nz, 15, 18)
    rhs = [rng.standard_normal(shape) for _ in range(3)]
    sol = [rng.standard_normal(shape) for _ in range(3)]
    out = _solve(gpulib, rhs, sol)
    for c in range(3):
        assert rel_l2(out[c], _reference(rhs[c], sol[c])) <= 1e-12, c


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_finite_stay_in_their_component(gpulib, bad):
    if gpulib.arith != "fp64":
        pytest.skip("the products are FP64's; float-float has no infinities or NaN")
    rng = np.random.default_rng(5)
    shape = (14, 102, 101)
    rhs = [rng.standard_normal(shape) for _ in range(3)]
    sol = [np.zeros(shape) for _ in range(3)]
    rhs[0][5, 40, 50] = bad
    out = _solve(gpulib, rhs, sol)
    assert not np.isfinite(out[0][1:-1, 1:-1, 1:-1]).any()
    for c in (1, 2):
        assert rel_l2(out[c], _reference(rhs[c], sol[c])) <= 1e-12
