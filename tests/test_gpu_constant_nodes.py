"""Samples over which nothing varies, for a plan whose quadrature nodes come in
descending order (the same integrator with its weights' columns reversed):
segments that end between the two nodes of a sample's first or last fine step
vary inside that sample, and every kernel that knows the maps gives the oracle's
states."""
import numpy as np
import pytest

from test_gpu_constant import _reference, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,lanes", [(0, 0), (6, 16), (6, 128), (7, 32), (8, 128)])
def test_descending_nodes(variant, lanes):
    from superspinsim_gb300 import _lib
    dt, T, F, B = 1e-10, 8, 8, 4
    c, vm, N, progs, rho, W, nodes, _, flat = _setup(0, 0, B=B)
    h = dt/F
    # pulses from inside the last fine step of sample 1 to inside the first of
    # sample 4, between the nodes at 0.21 and 0.79 of the step
    progs[:, 0, :, 0] = -np.inf
    progs[:, 0, 0] = (2*dt - 0.5*h, 0, 0, 0, 0)
    progs[:, 0, 1] = (4*dt + 0.5*h, 0, 1e-4, 3.1e9, 0.2)
    progs[:, 0, 2] = (np.inf, 0, 0, 0, 0)
    progs[:, 3, :, 0] = -np.inf
    progs[:, 3, 0] = (5*dt - 0.5*h, 0.15, 0, 0, 0)
    progs[:, 3, 1] = (np.inf, 0, 0, 0, 0)
    plan = _lib.Plan(c["generators"], np.ascontiguousarray(W[:, ::-1]), nodes[::-1].copy())
    plan.set_batch_config(lanes=lanes, variant=variant)
    _, _, tr = plan.batch(flat, progs, 0.0, dt, T, F, want_final=True, want_trace=True)
    ref = _reference(c, vm, progs, rho, W, nodes, 0.0, dt, T, F)
    assert np.abs(tr - ref).max() <= 1e-12
