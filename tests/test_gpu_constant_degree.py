"""A plan with a fixed Taylor degree steps the samples over which nothing varies
at that degree, like all others: at degree 1 (its sub-steps end at 1,024, so the
first order shows) every slot-programmed kernel agrees with the row-part kernel,
which knows no maps, and all of them miss the exact evolution."""
import numpy as np
import pytest

from test_gpu_constant import _reference, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,lanes", [(0, 0), (6, 16), (6, 128), (7, 32)])
def test_fixed_degree_steps_constant_samples(variant, lanes):
    from superspinsim_gb300 import _lib
    dt, T, F, B = 1e-10, 16, 8, 3
    c, vm, N, progs, rho, W, nodes, _, flat = _setup(0, 0, B=B)
    out = {}
    for v, ln in ((4, 32), (variant, lanes)):
        plan = _lib.Plan(c["generators"], W, nodes, taylor_degree=1)
        plan.set_batch_config(lanes=ln, variant=v)
        _, out[v] = plan.batch(flat, progs, 0.0, dt, T, F, want_final=True)
        info = plan.batch_info()
        assert info["degree"] == 1 and info["substeps"] == 1024
    # 262,144 sub-steps, each rounding the state once
    assert np.abs(out[variant] - out[4]).max() <= 1e-11
    exact = _reference(c, vm, progs, rho, W, nodes, 0.0, dt, T, F)[:, -1]
    assert np.abs(out[4] - exact).max() >= 1e-8
