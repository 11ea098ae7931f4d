"""The near field's plan (csrc/near_host.cpp) on the CPU: a restatement of the
kernel's products from the plan's tables and runs, with every index checked
against its array, equals the direct sum over the lattice rule (cells whose
parents are opened and that are not; the coarsest level's opened cells with
the opposite sign).  Both add the same FP64 weights in different orders:
n cells of similar size give n ulp at most, 1e-12 for the few thousand here.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan_program(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("near") / "near_plan_check")
    csrc = os.path.join(ROOT, "vpm_free_gb300", "csrc")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + csrc,
                    os.path.join(ROOT, "tests", "near_plan_check.cpp"), os.path.join(csrc, "near_host.cpp"), "-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("shape,h,levmax", [
    ((9, 13, 17), (0.1, 0.1, 0.1), 1),       # opposite faces within the opening radius; ties
    ((17, 25, 33), (0.1, 0.1, 0.1), 2),
    ((41, 41, 41), (0.1, 0.1, 0.1), 2),
    ((33, 25, 41), (0.1, 0.12, 0.09), 3),    # unequal spacings: tables of their own per pair of axes
    ((33, 65, 33), (0.05, 0.05, 0.07), 4),
])
def test_plan_equals_the_direct_sum(plan_program, shape, h, levmax):
    out = subprocess.run([plan_program, *map(str, shape), *map(str, h), str(levmax)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert float(out.stdout) <= 1e-12


@pytest.mark.parametrize("shape,levmax", [((27, 35, 30), 3), ((9, 17, 17), 3), ((18, 17, 17), 1)])
def test_ragged_lattices_have_no_plan(plan_program, shape, levmax):
    out = subprocess.run([plan_program, *map(str, shape), "0.1", "0.1", "0.1", str(levmax)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "no plan"
