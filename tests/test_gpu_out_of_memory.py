"""Set-up where one device allocation fails, by a preloaded cudaMalloc that says
so: the arrays of the boundary operator's FFT and tables are a choice of speed,
so define_sizes does without them, as it does without a recorded list, and the
solve stays the same."""
import json
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, json, os, sys
sys.path.insert(0, %r)
import numpy as np
import vpm_free_gb300 as V
shim = ctypes.CDLL(None)
cells, h = 32, 0.1
cfg = V.VPMConfig.make(dpm=(h,) * 3, box=(0, 0, 0) + (cells * h,) * 3)
rhs = np.random.default_rng(1).standard_normal((3,) + (cells + 1,) * 3)
x = np.full((1, 3), 0.5 * cells * h)
res = {}
for mode in ("1", "0"):
    os.environ["VPMG_FARFIELD"] = mode
    with V.VPM(cfg) as H:
        shim.malloc_fails_at(0)
        H.define_sizes(x)
        n = shim.malloc_calls()
        good, on = H.apply_poisson(rhs), H.farfield_stats()["on"]
    refused, without, worst = 0, 0, 0.0
    for k in range(1, n + 1):
        with V.VPM(cfg) as H:
            shim.malloc_fails_at(k)
            try:
                H.define_sizes(x)
            except V.VPMError as e:
                assert e.status == -3, e
                refused += 1
                continue
            finally:
                shim.malloc_fails_at(0)
            without += on and not H.farfield_stats()["on"]
            worst = max(worst, float(np.abs(H.apply_poisson(rhs) - good).max() / np.abs(good).max()))
    res[mode] = dict(on=on, calls=n, refused=refused, without=without, worst=worst)
print(json.dumps(res))
"""


def test_operator_without_room_for_its_tables(gpulib, tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc or gpulib.arith != "fp64":
        pytest.skip("no C compiler, or the second arithmetic")
    so = str(tmp_path / "cuda_malloc_fails.so")
    subprocess.run([cc, "-shared", "-fPIC", "-O1", os.path.join(ROOT, "tests", "cuda_malloc_fails.c"), "-o", so, "-ldl"],
                   check=True)
    out = subprocess.run([sys.executable, "-c", CHILD % ROOT], env=dict(os.environ, LD_PRELOAD=so), capture_output=True,
                         text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    r = json.loads(out.stdout)
    assert r["1"]["on"] and not r["0"]["on"]
    assert r["1"]["without"] >= 10, r               # each of its arrays in turn
    assert r["1"]["refused"] <= r["0"]["refused"], r  # the fields, plans and trees, which both need
    assert max(r["1"]["worst"], r["0"]["worst"]) <= 1e-13, r
