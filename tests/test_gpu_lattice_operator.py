"""The boundary operator of uniform lattices, the coarsest level by FFT and the
opened cells by weight tables (csrc/farfield.cu, csrc/nearfield.cu), against the
recorded rows of the same operator (VPMG_FARFIELD=0), through a handle's
vector-potential solve of seeded random right-hand sides.

Both sum the same weights in another order and rounding: the tables hold them to
2^-55 of the largest and the FFT adds a few units of 2^-53 per stage, so the
solutions agree to 1e-13 in FP64; float-float rows keep 48 bits of each weight
and source, 1e-12.
"""
import numpy as np
import pytest

from helpers import configs_for, rel_l2

pytestmark = pytest.mark.gpu


def _solve(V, monkeypatch, cells, h, tables, origin=(0.0, 0.0, 0.0), **cfg):
    if tables:
        monkeypatch.delenv("VPMG_FARFIELD", raising=False)
    else:
        monkeypatch.setenv("VPMG_FARFIELD", "0")
    h = np.broadcast_to(np.asarray(h, dtype=np.float64), 3)
    lo = np.asarray(origin, dtype=np.float64)
    box = tuple(lo) + tuple(lo + np.asarray(cells) * h)
    with V.VPM(V.VPMConfig.make(dpm=tuple(h), box=box, **cfg)) as H:
        H.define_sizes(np.array([lo + 0.5 * np.asarray(cells) * h]))
        r = np.random.default_rng(5).standard_normal(tuple(H._mesh_shape()))
        return H.apply_poisson(r), H.farfield_stats()["on"]


def _same(gpulib, monkeypatch, cells, h, **kw):
    a, on = _solve(gpulib, monkeypatch, cells, h, True, **kw)
    b, off = _solve(gpulib, monkeypatch, cells, h, False, **kw)
    assert on and not off
    for c in range(3):
        assert rel_l2(a[c], b[c]) <= (1e-13 if gpulib.arith == "fp64" else 1e-12), (c, rel_l2(a[c], b[c]))


# 48^3 cells: 25 thousand boundary nodes of the padded block; 96^3: 75 thousand,
# where float-float handles take the tables too
@pytest.mark.parametrize("h", [1.3e-5, 1e-5, 1e-6, 1.25e-7, 1e-8])
def test_spacings_below_the_panel_distance(gpulib, monkeypatch, h):
    """Cells within 1e-5 of a node weigh as a panel at its own centre: the nearest
    leaf cells at 1.3e-5, whole levels below (distances of exactly 1e-5 among
    them), and accepted coarsest cells at 1e-7 and less."""
    if gpulib.arith != "fp64" and h != 1e-6:
        pytest.skip("one spacing in float-float")
    _same(gpulib, monkeypatch, (48,) * 3 if gpulib.arith == "fp64" else (96,) * 3, h)


@pytest.mark.parametrize("spacings,on", [(1e4, True), (1e6, False)])
def test_boxes_far_from_the_origin(gpulib, monkeypatch, spacings, on):
    """Coordinates rounded to 1e-10 of a spacing decide weights of their own: such
    boxes keep the walk's (tests/test_lattice_origin.py has the limit)."""
    if gpulib.arith != "fp64":
        pytest.skip("float-float handles of this size record")
    org = (0.05 * spacings * 1.0000001,) * 3
    got, tables = _solve(gpulib, monkeypatch, (48, 48, 48), 0.05, True, origin=org)
    assert tables == on
    rows, _ = _solve(gpulib, monkeypatch, (48, 48, 48), 0.05, False, origin=org)
    for c in range(3):
        assert rel_l2(got[c], rows[c]) <= (1e-13 if on else 0.0), c


@pytest.mark.parametrize("cells,thin", [((64, 64, 64), 80), ((48, 24, 56), 40), ((64, 48, 32), 80)])
def test_faces_exactly_an_opening_radius_apart(gpulib, monkeypatch, cells, thin):
    """At a spacing of 1/64 the sides' distance (80 or 40 spacings of the padded
    block) is exactly ten cell sides of some level: no cell is opened across,
    and the table of that pair of faces is empty."""
    if gpulib.arith != "fp64":
        pytest.skip("float-float handles of this size record")
    assert any(c + 16 == thin for c in cells)
    _same(gpulib, monkeypatch, cells, 1.0 / 64)


# cells, spacings, ilevmax, ncoarse: three different sides (FFT lengths with and without radix 3), unequal
# spacings (tables of their own for every pair of axes), two and four levels
BOXES = [((40, 56, 48), (0.05, 0.05, 0.05), 3, 8),
         ((64, 48, 40), (0.025, 0.04, 0.03), 3, 8),
         ((36, 52, 44), (0.06, 0.05, 0.07), 2, 4),
         ((64, 48, 80), (0.05, 0.05, 0.06), 4, 8),
         ((104, 88, 96), (0.03, 0.04, 0.025), 3, 8)]


@pytest.mark.parametrize("cells,h,levmax,ncoarse", BOXES)
def test_tables_equal_recorded_rows(gpulib, monkeypatch, cells, h, levmax, ncoarse):
    if gpulib.arith != "fp64" and cells[0] < 100:
        pytest.skip("float-float handles record below 60 thousand boundary nodes")
    _same(gpulib, monkeypatch, cells, h, ilevmax=levmax, ncoarse=ncoarse)


@pytest.mark.parametrize("cells,h,levmax", [((40, 56, 48), (0.05, 0.05, 0.05), 3), ((40, 48, 32), (0.06, 0.05, 0.075), 2)])
def test_tables_in_a_step_equal_the_oracle(gpulib, oracle, monkeypatch, cells, h, levmax):
    """A whole field step of random particles on boxes of unequal sides and
    spacings: the mesh fields within 1e-10 of the oracle's."""
    if gpulib.arith != "fp64":
        pytest.skip("float-float handles of this size record")
    monkeypatch.delenv("VPMG_FARFIELD", raising=False)
    V, O = gpulib, oracle
    L = np.asarray(cells) * h
    rng = np.random.default_rng(8)
    n = 2000
    xp = np.ascontiguousarray(L / 2 + rng.uniform(-0.3, 0.3, (n, 3)) * L)
    qp = np.concatenate([rng.normal(0, 1e-3, (n, 3)), np.full((n, 1), np.prod(h))], 1)
    ocfg, gcfg = configs_for(dict(dpm=tuple(h), box=(0.0, 0.0, 0.0) + tuple(L)), ilevmax=levmax)
    s = O.define_sizes(ocfg, xp)
    O.step_fields(ocfg, s, xp, qp)
    with V.VPM(gcfg) as H:
        H.define_sizes(xp)
        assert H.farfield_stats()["on"]
        up, gp = np.zeros((n, 3)), np.zeros((n, 3))
        H.vpm(xp, qp, up, gp, n, WhatToDo=2)
        for name, fid in (("sol", O.F_SOL), ("vel", O.F_VEL), ("def", O.F_DEF)):
            assert rel_l2(H.field(name).ravel(), O.get_field(fid)) <= 1e-10, name


def test_large_pmesh_takes_the_tables(gpulib, monkeypatch):
    """pmesh from 100 thousand boundary nodes on goes by FFT and tables, below by one
    walk: 145 x 129 x 137 nodes (112 thousand) against the walk that VPMG_FARFIELD=0 leaves."""
    shape, h = (137, 129, 145), (0.05, 0.04, 0.06)
    nz, ny, nx = shape
    rng = np.random.default_rng(4)
    rhs = [rng.standard_normal(shape) for _ in range(3)]
    xb = (0.0, 0.0, 0.0, (nx - 1) * h[0], (ny - 1) * h[1], (nz - 1) * h[2])
    out = []
    for env in (None, "0"):
        if env is None:
            monkeypatch.delenv("VPMG_FARFIELD", raising=False)
        else:
            monkeypatch.setenv("VPMG_FARFIELD", env)
        sol = [np.zeros(shape) for _ in range(3)]
        with gpulib.VPM(gpulib.VPMConfig.make(dpm=h, box=(0, 0, 0) + tuple(8 * v for v in h))) as H:
            H.pmesh(sol, rhs, xb, h, iynbc=1, itree=1, levmax=3)
        out.append(sol)
    # the walk adds its cells one by one: some thousand terms, 1e-12
    for c in range(3):
        assert rel_l2(out[0][c], out[1][c]) <= 1e-12, c
        assert not np.array_equal(out[0][c], out[1][c])
