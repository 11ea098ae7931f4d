"""A handle that is sized anew, as the reference's define_sizes does for new
particles: captured steps of the mesh that was are not replayed, and a batch
whose shared operator belonged to it says so."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(scale):
    from vpm_free_gb300 import workloads as W
    xp, qp, w = W.scaled_ring(32)
    return np.ascontiguousarray(scale * xp), qp, w


def _advance(h, xp, qp, dt):
    h.define_sizes(xp)
    h.set_particles(xp, qp)
    h.run(2, dt)
    return h.get_particles()


def test_run_after_define_sizes(gpulib):
    V = gpulib
    x1, q1, w = _ring(1.0)
    x2, q2, _ = _ring(1.4)
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"])) as h:
        _advance(h, x1, q1, w["dt"])
        n1 = list(h.sizes().nn)
        again = _advance(h, x2, q2, w["dt"])
        assert list(h.sizes().nn) != n1
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"])) as h:
        fresh = _advance(h, x2, q2, w["dt"])
    for a, b in zip(again, fresh):
        assert np.array_equal(a, b)


def test_new_arrays_hold_no_particles(gpulib):
    """Before set_particles, and after a mesh that needs larger arrays."""
    V = gpulib
    x1, q1, w = _ring(1.0)
    x2, _, _ = _ring(1.4)
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"])) as h:
        for x in (x1, x2):
            h.define_sizes(x)
            assert h.num_particles() == 0
            h.run(1, w["dt"])
            assert h.get_particles()[0].shape[0] == 0
            h.set_particles(x1, q1)


def test_gradient_after_define_sizes(gpulib):
    if gpulib.arith != "fp64":
        pytest.skip("one arithmetic")
    V = gpulib
    x1, q1, w = _ring(1.0)
    x2, q2, _ = _ring(1.4)

    def grad(h, xp, qp):
        h.define_sizes(xp)
        h.set_particles(xp, qp)
        return h.adjoint_run(2, w["dt"], ke_weight=0.1)[:3]
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"])) as h:
        grad(h, x2, q2)
        grad(h, x1, q1)  # the smaller mesh fits the larger one's arrays
        again = grad(h, x2, q2)
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"])) as h:
        fresh = grad(h, x2, q2)
    assert abs(again[0] - fresh[0]) <= 1e-13 * abs(fresh[0])
    for a, b in zip(again[1:], fresh[1:]):  # sums by atomics, in any order
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()


def test_batch_after_define_sizes(gpulib, monkeypatch):
    monkeypatch.setenv("VPMG_FARFIELD", "0")  # recorded operators are shared
    V = gpulib
    x1, q1, w = _ring(1.0)
    x2, q2, _ = _ring(1.4)
    hs = [V.VPM(V.VPMConfig.make(dpm=w["dpm"])) for _ in range(2)]
    for h in hs:
        h.define_sizes(x1)
        h.set_particles(x1, q1)
    with V.Batch(hs) as b:
        assert b.info() == (1, 2)
        b.run(1, w["dt"])
        hs[1].define_sizes(x2)
        hs[1].set_particles(x2, q2)
        with pytest.raises(V.VPMError) as e:
            b.run(1, w["dt"])
        assert e.value.status == -7
    with V.Batch(hs) as b:
        b.run(1, w["dt"])
    for h in hs:
        h.close()
