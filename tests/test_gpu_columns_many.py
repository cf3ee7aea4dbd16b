"""Drop-in runs of more trajectories than a grid's y dimension has blocks
(65,535): the trajectories around the boundary agree with the same ones run as a
small batch and with the oracle, and the rest lie between their neighbours.  Lab
frame and rotating frame (whose states pass through one more kernel)."""
import numpy as np
import pytest

from conftest import load_case
from oracle import oracle
from test_gpu_columns import _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rot", [False, True])
@pytest.mark.parametrize("B,T", [(65536, 1), (70000, 2)])
def test_more_trajectories_than_grid_rows(B, T, rot):
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    dt, F = 1e-10, 2
    plan, W, nodes = _plan(c, 2, dt, F, rot, True)
    progs = np.zeros((B, 4, 1, 5))
    progs[..., 0] = np.inf
    amp = 1e-4*np.linspace(0.5, 1, B)
    progs[:, 0, 0, 2] = amp
    progs[:, 0, 0, 3] = 2.9e9
    rho = np.diag([0.25, 0.75, 0.0]).astype(complex)
    flat = oracle.flatten(rho, vm, N)
    out = plan.simulate(np.stack([flat]*B), progs, 0.0, dt, T, F)
    pick = np.array([0, 1, 65533, 65534, 65535, B - 1])
    small = plan.simulate(np.stack([flat]*pick.size), progs[pick], 0.0, dt, T, F)
    # the lane rule may deal few trajectories other lanes than many: the same
    # sums in another order (the eigenbasis costs its condition number, below 100)
    assert np.abs(out[pick] - small).max() <= (1e-12 if rot else 1e-14)
    # neighbours differ by their drives: at most |G_x| da t on a state of 1-norm below 4
    step = np.abs(c["generators"][1]).sum(0).max()*(amp[1] - amp[0])*T*dt
    assert np.abs(np.diff(out[:, -1], axis=0)).max() <= 4*step + 1e-12
    if not rot:
        _, ref = oracle.simulate(c["generators"], np.stack([rho]*pick.size), 0.0, T*dt + 1e-14, dt,
                                 progs[pick], K=2, W=W, nodes=nodes, F=F, vectorisation_map=vm,
                                 mode="vector", degree=20, flat_out=True)
        assert np.abs(out[pick] - ref).max() <= 1e-12
