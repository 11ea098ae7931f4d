"""How far from zero a box may lie for its boundary operator to go by lattice
offsets (lattice_exact in csrc/near_host.cpp): the weights of the nearest cells
stay within 1e-10, the parity bar of the fields, of those that the quadtree walk
forms from rounded coordinates.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("origin") / "lattice_origin_check")
    csrc = os.path.join(ROOT, "vpm_free_gb300", "csrc")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + csrc,
                    os.path.join(ROOT, "tests", "lattice_origin_check.cpp"), os.path.join(csrc, "near_host.cpp"), "-o",
                    exe], check=True)
    return exe


@pytest.mark.parametrize("h", [0.05, 2.0 / 384, 0.0117187, 1.0 / 64])
@pytest.mark.parametrize("spacings", [0.0, 1e2, 1e4, 1e5, 2e5, 3e5, 5e5, 1e6, 3e6])
def test_accepted_boxes_keep_the_weights(program, h, spacings):
    x0 = -h * spacings * 1.0000001
    out = subprocess.run([program, "145", repr(h), repr(x0)], capture_output=True, text=True, check=True).stdout.split()
    accepted, worst = out[0] == "1", float(out[1])
    if spacings <= 1e4:
        assert accepted
    if worst > 1e-10:
        assert not accepted
    if accepted:
        assert worst <= 1e-10
