"""Bounded waits of the tensor-core kernels that run out: the call reports an
error (or, without a handle, returns NaN), never finite wrong values, and the
device stays usable.

VPMG_WAIT_POLLS sets how often a wait polls before it gives up: 0 makes every
wait run out with copies in flight, a few polls make some of them do so midway.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D = (0.05, 0.06, 0.04)
SHAPE = (82, 103, 101)  # products along x (N = 100) and y (N = 102), also for one component (126 and 124 tiles)


def _pmesh(V, rhs, sol):
    with V.VPM(V.VPMConfig.make(dpm=D, box=(0, 0, 0, 0.4, 0.48, 0.32))) as h:
        out = [s.copy() for s in sol]
        h.pmesh(out, rhs, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), D, iynbc=0, NN_bl=(1, 1, 1) + SHAPE[::-1])
    return out


@pytest.fixture
def fields():
    rng = np.random.default_rng(9)
    return ([rng.standard_normal(SHAPE) for _ in range(3)], [rng.standard_normal(SHAPE) for _ in range(3)])


@pytest.mark.parametrize("polls", [0, 1, 3, 10])
def test_product_passes_report_waits_that_run_out(gpulib, monkeypatch, fields, polls):
    if gpulib.arith != "fp64":
        pytest.skip("the products are FP64's")
    V = gpulib
    good = _pmesh(V, *fields)
    monkeypatch.setenv("VPMG_WAIT_POLLS", str(polls))
    try:
        got = _pmesh(V, *fields)
        assert polls > 0
        assert all(np.array_equal(a, b) for a, b in zip(got, good))
    except V.VPMError as e:
        assert e.status == -2 and "wait" in str(e)
    monkeypatch.delenv("VPMG_WAIT_POLLS")
    assert all(np.array_equal(a, b) for a, b in zip(_pmesh(V, *fields), good))


def test_static_solve_shows_nan(gpulib, monkeypatch, fields):
    torch = pytest.importorskip("torch")
    f = gpulib.load_library().vpmg_dirichlet_static
    f.argtypes = [C.c_void_p, C.c_void_p, C.POINTER(C.c_int), C.POINTER(C.c_int), C.POINTER(C.c_double), C.c_int,
                  C.c_void_p]
    a = torch.from_numpy(fields[0][0]).cuda()
    nx, ny, nz = SHAPE[::-1]

    def solve():
        b = torch.from_numpy(fields[1][0]).cuda()
        assert f(a.data_ptr(), b.data_ptr(), (C.c_int * 3)(nx, ny, nz), (C.c_int * 6)(0, 0, 0, nx - 1, ny - 1, nz - 1),
                 (C.c_double * 3)(*D), 0, None) == 0
        torch.cuda.synchronize()
        return b.cpu().numpy()
    good = solve()
    monkeypatch.setenv("VPMG_WAIT_POLLS", "0")
    assert np.isnan(solve()[1:-1, 1:-1, 1:-1]).all()
    monkeypatch.delenv("VPMG_WAIT_POLLS")
    assert np.array_equal(solve(), good)


def test_steps_report_waits_that_run_out(gpulib, monkeypatch):
    """A driver call and the captured step of a 96^3 ring (lines of N = 112)."""
    from vpm_free_gb300 import workloads as W
    if gpulib.arith != "fp64":
        pytest.skip("the products are FP64's")
    V = gpulib
    xp, qp, w = W.scaled_ring(96)
    cfg = V.VPMConfig.make(dpm=w["dpm"], box=w["box"])
    n = xp.shape[0]
    monkeypatch.setenv("VPMG_WAIT_POLLS", "0")
    with V.VPM(cfg) as h:
        h.define_sizes(xp)
        up, gp = np.zeros((n, 3)), np.zeros((n, 3))
        with pytest.raises(V.VPMError, match="wait"):
            h.vpm(xp, qp, up, gp, n, WhatToDo=2)
        h.set_particles(xp, qp)
        with pytest.raises(V.VPMError, match="wait"):
            h.run(1, 0.01)
    monkeypatch.delenv("VPMG_WAIT_POLLS")
    with V.VPM(cfg) as h:
        h.define_sizes(xp)
        up, gp = np.zeros((n, 3)), np.zeros((n, 3))
        h.vpm(xp, qp, up, gp, n, WhatToDo=2)
        assert np.isfinite(up).all() and np.isfinite(gp).all()


@pytest.mark.parametrize("polls", [0, 1, 3, 10])
def test_boundary_operator_reports_waits_that_run_out(gpulib, monkeypatch, polls):
    """The weight tables' products (81^3 block of the 64^3 ring, 113^3 in
    float-float; the lines of the former go by FFT)."""
    from vpm_free_gb300 import workloads as W
    V = gpulib
    xp, qp, w = W.ring64() if gpulib.arith == "fp64" else W.scaled_ring(96)
    cfg = V.VPMConfig.make(dpm=w["dpm"], box=w["box"])
    n = xp.shape[0]

    def step():
        with V.VPM(cfg) as h:
            h.define_sizes(xp)
            assert h.farfield_stats()["on"]
            up, gp = np.zeros((n, 3)), np.zeros((n, 3))
            h.vpm(xp, qp, up, gp, n, WhatToDo=2)
            return up
    good = step()
    monkeypatch.setenv("VPMG_WAIT_POLLS", str(polls))
    try:
        got = step()
        assert polls > 0 and np.array_equal(got, good)
    except V.VPMError as e:
        assert e.status == -2 and "wait" in str(e)
    monkeypatch.delenv("VPMG_WAIT_POLLS")
    assert np.array_equal(step(), good)
