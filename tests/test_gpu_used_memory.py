"""Results do not depend on what device memory held before: every entry point on
memory that was filled with NaN and given back gives the bits it gave on fresh
memory.  The coarse grids have dummy tree cells (14 and 13 cells a side at two
levels), whose sources nothing writes.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _UsedMemory:
    """Blocks of many sizes filled with NaN and given back; every eighth is kept, so
    that the chunks they came from stay with the process."""

    def __init__(self):
        self.rt = C.CDLL("libcudart.so.13")  # the library's own
        self.rt.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
        self.rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
        self.rt.cudaFree.argtypes = [C.c_void_p]
        nan = np.full(1 << 17, np.nan)
        got = []
        for size in (1 << 12, 1 << 14, 1 << 15, 1 << 16, 1 << 18, 1 << 20):
            for _ in range(96):
                got.append(self._block(size))
                assert self.rt.cudaMemcpy(got[-1], nan.ctypes.data, size, 1) == 0
        self.kept = got[::8]
        for q in set(q.value for q in got) - set(q.value for q in self.kept):
            assert self.rt.cudaFree(q) == 0

    def _block(self, size):
        q = C.c_void_p()
        assert self.rt.cudaMalloc(C.byref(q), size) == 0
        return q

    def comes_back(self):
        """Whether a new block holds what a freed one held."""
        host = np.zeros(1 << 11)
        q = self._block(host.nbytes)
        assert self.rt.cudaMemcpy(host.ctypes.data, q, host.nbytes, 2) == 0
        assert self.rt.cudaFree(q) == 0
        return bool(np.isnan(host).any())

    def close(self):
        for q in self.kept:
            self.rt.cudaFree(q)


@pytest.fixture
def used_memory():
    made = []

    def use():
        made.append(_UsedMemory())
        if not made[0].comes_back():
            pytest.skip("freed device memory does not come back as it was")
    yield use
    for m in made:
        m.close()


def _step(V):
    from vpm_free_gb300 import workloads as W
    xp, qp, w = W.scaled_ring(48)
    with V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
        h.define_sizes(xp)
        up, gp = np.zeros_like(xp), np.zeros_like(xp)
        h.vpm(xp, qp, up, gp, xp.shape[0], WhatToDo=2)
        h.set_particles(xp, qp)
        h.run(2, w["dt"])
        return (up, gp) + tuple(h.get_particles())


def _coarse(V):
    """40 x 40 x 48 cells with the panel boundary, several blocks, two levels."""
    out = []
    for kw in (dict(ibctyp=3), dict(nb=(1, 1, 2)), dict(ilevmax=2), dict(ncoarse=4), dict(iyntree=0)):
        c = (24, 24, 32) if "iyntree" in kw else (40, 40, 48)
        with V.VPM(V.VPMConfig.make(dpm=(0.05,) * 3, box=(0.0, 0.0, 0.0) + tuple(0.05 * k for k in c), **kw)) as h:
            h.define_sizes(np.array([[0.6, 0.6, 0.7]]))
            r = np.random.default_rng(1).standard_normal(tuple(h._mesh_shape()))
            out.append(h.apply_poisson(r))
    return out


def _pmesh(V):
    out = []
    for shape, lev in (((27, 35, 30), 3), ((33, 25, 29), 2)):
        rhs = [np.random.default_rng(2 + c).standard_normal(shape) for c in range(3)]
        sol = [np.zeros(shape) for _ in range(3)]
        nz, ny, nx = shape
        with V.VPM(V.VPMConfig.make(dpm=(0.1,) * 3, box=(0.0, 0.0, 0.0, 0.8, 0.8, 0.8))) as h:
            h.pmesh(sol, rhs, (0.0, 0.0, 0.0, 0.1 * (nx - 1), 0.1 * (ny - 1), 0.1 * (nz - 1)), (0.1,) * 3, iynbc=1,
                    itree=1, levmax=lev)
        out += sol
    return out


def _batch(V):
    from vpm_free_gb300 import workloads as W
    hs, out = [], []
    for k in range(3):
        xp, qp, w = W.scaled_ring((32, 32, 48)[k])
        h = V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"]))
        h.define_sizes(xp)
        h.set_particles(xp, qp)
        hs.append(h)
    with V.Batch(hs) as b:
        b.set_schedule(1)
        b.run(2, 0.01)
    for h in hs:
        out += list(h.get_particles())
        h.close()
    return out


@pytest.mark.parametrize("call", [_step, _coarse, _pmesh, _batch])
def test_bits_do_not_depend_on_used_memory(gpulib, used_memory, call):
    first = call(gpulib)
    used_memory()
    for a, b in zip(first, call(gpulib)):
        assert np.isfinite(b).all()
        assert np.array_equal(a, b)


def test_gradient_does_not_depend_on_used_memory(gpulib, used_memory):
    from vpm_free_gb300 import workloads as W
    xp, qp, w = W.scaled_ring(48)

    def grad():
        with gpulib.VPM(gpulib.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
            h.define_sizes(xp)
            h.set_particles(xp, qp)
            return h.adjoint_run(2, w["dt"], probes=np.array([[0.3, 0.2, 0.1]]), ke_weight=0.1)[:3]
    first = grad()
    used_memory()
    for a, b in zip(first, grad()):  # position gradients add by atomics, in any order
        assert np.abs(np.asarray(a) - np.asarray(b)).max() <= 1e-10 * np.abs(np.asarray(a)).max()
