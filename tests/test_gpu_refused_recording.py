"""Gradients of an operator whose interaction list does not fit the budget: the
list is counted and refused once, on the first call, not on every one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_refused_list_is_not_counted_again(gpulib):
    from vpm_free_gb300 import workloads as W
    if gpulib.arith != "fp64":
        pytest.skip("float-float handles of this size record in define_sizes")
    V = gpulib
    xp, qp, w = W.ring64()
    launches, loss = {}, {}
    for name, budget in (("fits", None), ("refused", 400 << 20)):
        with V.VPM(V.VPMConfig.make(dpm=w["dpm"], box=w["box"])) as h:
            if budget:
                h.set_operator_budget(budget)
            h.define_sizes(xp)
            assert h.farfield_stats()["on"] and not h.tree_stats()["precomputed"]
            h.set_particles(xp, qp)
            got = []
            for _ in range(3):  # a loss alone: prepares the transposes, launches none
                l0 = h.kernel_launches()
                loss[name] = h.adjoint_loss(1, w["dt"], ke_weight=0.1)
                got.append(h.kernel_launches() - l0)
            assert h.tree_stats()["precomputed"] == (budget is None)
            launches[name] = got
            if budget:  # walked transposes, before and after
                g = [h.adjoint_run(1, w["dt"], ke_weight=0.1)[2] for _ in range(2)]
                assert np.allclose(g[0], g[1], rtol=0, atol=1e-12 * np.abs(g[0]).max())
    assert launches["fits"][1] == launches["fits"][2]
    assert launches["refused"][1:] == launches["fits"][1:], launches
    assert launches["refused"][0] > launches["refused"][1]
    assert loss["fits"] == loss["refused"]
