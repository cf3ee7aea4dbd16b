"""The smallest drop-in calls take dense propagators (two launches), larger ones
columns (three and more): both sides of the rule's edges in samples, exponentials,
trajectories and rows, in both frames, against the oracle or each other; and
columns of exponents so large that the Taylor action takes sub-steps."""
import numpy as np
import pytest

from conftest import load_case
from oracle import oracle
from test_gpu_columns import _plan

pytestmark = pytest.mark.gpu


def _run(name, B, T, F, K, rot, dt=1e-10):
    c = load_case(name)
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    n = int(vm[:, 0].max()) + 1
    plan, W, nodes = _plan(c, K, dt, F, rot, True)
    rng = np.random.default_rng(T)
    progs = np.zeros((B, 4, 1, 5))
    progs[..., 0] = np.inf
    progs[:, 0, 0, 2] = 1e-4*rng.uniform(0.5, 1, B)
    progs[:, 0, 0, 3] = 2.9e9
    rho = np.zeros((n, n), complex)
    rho[1, 1], rho[0, 0] = 0.75, 0.25
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    out = plan.simulate(flat, progs, 0.0, dt, T, F)
    ref = None
    if not rot:
        _, ref = oracle.simulate(c["generators"], np.stack([rho]*B), 0.0, T*dt + dt/4, dt, progs,
                                 K=K, W=W, nodes=nodes, F=F, vectorisation_map=vm, mode="vector",
                                 degree=20, flat_out=True)
    return plan, out, ref


@pytest.mark.parametrize("B,T,F,K,dense", [(1, 1, 1, 1, True), (1, 32, 5, 1, True), (1, 32, 1, 5, True),
                                           (1, 33, 5, 1, False), (1, 32, 6, 1, False),
                                           (1, 3, 3, 2, False), (2, 3, 1, 1, False)])
def test_edges_of_the_small_calls(B, T, F, K, dense):
    plan, out, ref = _run("spin1_c1", B, T, F, K, False)
    assert (plan.last_launches() == 2) == dense
    assert np.abs(out - ref).max() <= 1e-12
    plan, _, _ = _run("spin1_c1", B, T, F, K, True)
    assert (plan.last_launches() == 2) == dense


def test_both_paths_in_the_rotating_frame():
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    plan, _, _ = _plan(c, 2, 1e-10, 2, True, True)
    prog = np.zeros((1, 4, 1, 5))
    prog[..., 0] = np.inf
    prog[0, 0, 0, 2:4] = (1e-4, 2.9e9)
    flat = oracle.flatten(np.diag([0.25, 0.75, 0.0]).astype(complex), vm, vm.shape[0])[None]
    short = plan.simulate(flat, prog, 0.0, 1e-10, 32, 2)
    assert plan.last_launches() == 2
    long = plan.simulate(flat, prog, 0.0, 1e-10, 33, 2)
    assert plan.last_launches() > 2
    # the eigenbasis costs its condition number (below 100) in rounding
    assert np.abs(long[:, :32] - short).max() <= 1e-11


@pytest.mark.parametrize("dt", [6e-9, 6e-8])
def test_columns_of_large_exponents(dt):
    """Six fine steps of 1 and 10 ns per sample under a constant field: exponents
    of norm 20 and 200, on columns by sub-steps or, beyond their range, dense."""
    from scipy.linalg import expm
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    plan, _, _ = _plan(c, 1, dt, 6, False, True)
    prog = np.zeros((1, 4, 1, 5))
    prog[..., 0] = np.inf
    prog[0, 0, 0, 1] = 1e-4
    flat = oracle.flatten(np.diag([0.25, 0.75, 0.0]).astype(complex), vm, vm.shape[0])
    out = plan.simulate(flat[None], prog, 0.0, dt, 3, 6)[0]
    L = (c["generators"][0] + 1e-4*c["generators"][1])*dt/6
    x, E = flat, np.linalg.matrix_power(expm(L), 6)
    for t in range(3):
        x = E @ x
        assert np.abs(out[t] - x).max() <= 6*(1e-12 + 64*2.0**-53*np.abs(L).sum(0).max())
