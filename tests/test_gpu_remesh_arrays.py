"""remesh_particles_3d over the forms of its host arrays: the contiguous ones go
up directly, the others through the handle's buffers; same particles (the same
kernels on the same values), same refusals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(V):
    d = (0.1, 0.1, 0.1)
    h = V.VPM(V.VPMConfig.make(dpm=d, box=(0.0, 0.0, 0.0, 1.6, 1.6, 1.6)))
    rng = np.random.default_rng(3)
    xp = 0.8 + 0.25 * rng.standard_normal((500, 3)).clip(-1.5, 1.5)
    qp = np.concatenate([rng.standard_normal((500, 3)), np.full((500, 1), 1e-3)], axis=1)
    h.define_sizes(xp)
    return h, xp, qp


def test_array_forms_give_the_same_particles(gpulib):
    h, xp, qp = _handle(gpulib)
    with h:
        x0, q0 = h.remesh_particles_3d(1, xp, qp)
        forms = [(np.asfortranarray(xp), qp), (xp, np.asfortranarray(qp)), (xp[::-1][::-1], qp),
                 (xp, np.concatenate([qp, qp[:7]]))]
        for x, q in forms:
            x1, q1 = h.remesh_particles_3d(1, x, q)
            assert np.array_equal(x1, x0) and np.array_equal(q1, q0)
            assert x1.flags.writeable and x1.shape[1] == 3 and q1.shape[1] == 4
        x2, q2 = h.remesh_particles_3d(1, np.empty((0, 3)), np.empty((0, 4)))
        assert x2.shape == (0, 3) and q2.shape == (0, 4)


def test_refusals(gpulib):
    V = gpulib
    h, xp, qp = _handle(V)
    with h:
        n = h.remesh_particles_3d(1, xp, qp)[0].shape[0]
        for x, q in ((xp, qp), (np.asfortranarray(xp), qp)):
            with pytest.raises(V.VPMError) as e:
                h.remesh_particles_3d(1, x, q, capacity=max(n - 1, x.shape[0]))
            assert e.value.status == -5
            with pytest.raises(V.VPMError) as e:
                h.remesh_particles_3d(2, x, q)
            assert e.value.status == -6
