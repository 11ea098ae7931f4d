"""Particles and probes far outside the mesh, beyond what a cell index can hold
among them, are refused with a status before anything is read or written there.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAR = [1e3, 1e9, 2147483646.0, 2147483648.0 * 0.1, 1e30, 1e300, np.inf, -1e30, -np.inf, np.nan]


def _ring():
    from vpm_free_gb300 import workloads as W
    xp, qp, w = W.scaled_ring(32)
    return xp, qp, w


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("far", FAR)
def test_particles(gpulib, axis, far):
    V = gpulib
    xp, qp, w = _ring()
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
        h.define_sizes(xp)
        up, gp = np.zeros_like(xp), np.zeros_like(xp)
        h.vpm(xp, qp, up, gp, xp.shape[0], WhatToDo=2)
        good = up.copy()
        bad = xp.copy()
        bad[7, axis] = far
        for call in (lambda: h.vpm(bad, qp, np.zeros_like(xp), np.zeros_like(xp), xp.shape[0], WhatToDo=2),
                     lambda: h.remesh_particles_3d(1, bad, qp),
                     lambda: (h.set_particles(bad, qp), h.run(1, w["dt"]))):
            with pytest.raises(V.VPMError) as e:
                call()
            assert e.value.status == -4
        up[:] = 0.0
        h.vpm(xp, qp, up, gp, xp.shape[0], WhatToDo=2)
        assert np.array_equal(up, good)


@pytest.mark.parametrize("far", FAR)
def test_probes(gpulib, far):
    V = gpulib
    xp, qp, w = _ring()
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
        h.define_sizes(xp)
        h.set_particles(xp, qp)
        with pytest.raises(V.VPMError) as e:
            h.adjoint_loss(1, w["dt"], probes=np.array([[0.1, 0.2, 0.3], [0.0, far, 0.0]]))
        assert e.value.status == -1
        assert np.isfinite(h.adjoint_loss(1, w["dt"], probes=np.array([[0.1, 0.2, 0.3]])))


def test_a_velocity_beyond_the_floats(gpulib):
    """Strengths whose velocities overflow: float-float's largest numbers are finite,
    and the Euler push takes the particles there."""
    V = gpulib
    xp, qp, w = _ring()
    q = qp.copy()
    q[:, :3] *= 1e36 if V.arith == "ff48" else 1e300
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
        h.define_sizes(xp)
        h.set_particles(xp, q)
        with pytest.raises(V.VPMError) as e:
            h.run(2, 1e6)
        assert e.value.status in (-4, -5)
        h.set_particles(xp, qp)
        h.run(1, w["dt"])
        assert np.isfinite(h.get_particles()[0]).all()
