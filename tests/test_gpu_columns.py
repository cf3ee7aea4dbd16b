"""Drop-in runs by propagator columns (sss_simulate from host buffers)
against the oracle, at the edges of the chain's blocks (16 samples) and of
the runs a column covers: lab and rotating frame, residual and plain
arithmetic, one and several coefficient tables, programs and sampled
coefficients, several trajectories, and a run so long that a column covers
several samples."""
import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


def _plan(c, K, dt, F, rot, res):
    from superspinsim_gb300 import _lib
    from superspinsim_gb300.generate_simulator import rotating_tables
    from superspinsim_gb300.rotating import make_rotating
    W, nodes = quadrature(K)
    gens = c["generators"]
    if not rot:
        return _lib.Plan(gens, W, nodes, residual=res), W, nodes
    new, V, Vi, d, s = make_rotating(gens[0], list(gens[1:]))
    gn, dl, sl = rotating_tables(np.array(new), d, s, nodes, dt/F, res)
    return _lib.Plan(None, W, nodes, residual=res,
                     rotating=dict(generators_nodes=gn, doubles_last=dl, singles_last=sl,
                                   vectors_real=V, inv_vectors_real=Vi)), W, nodes


def _programs(B, rng, amp):
    p = np.zeros((B, 4, 2, 5))
    p[:, :, 0, 0] = 7.3e-10
    p[:, :, 1, 0] = np.inf
    p[:, 0, :, 2] = amp*rng.uniform(0.5, 1, (B, 2))
    p[:, 0, :, 3] = 2.9e9*rng.uniform(0.9, 1.1, (B, 2))
    p[:, 0, :, 4] = rng.uniform(0, 6, (B, 2))
    return p


@pytest.mark.parametrize("T", [1, 15, 16, 17, 33, 70])
@pytest.mark.parametrize("name,K,rot,res", [("spin1_c1", 2, False, True), ("spin1_c1", 5, False, True),
                                            ("spin1_c1", 1, False, False), ("spin1_c1", 2, True, True),
                                            ("spin1_c1", 5, True, False), ("nv7_n49", 2, False, True),
                                            ("nv7_n49", 2, True, True)])
def test_columns_against_oracle(name, K, rot, res, T):
    c = load_case(name)
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    n = int(vm[:, 0].max()) + 1
    rng = np.random.default_rng(T)
    dt, F, B = 1e-10, 7, 2
    plan, W, nodes = _plan(c, K, dt, F, rot, res)
    progs = _programs(B, rng, 1e-4)
    if n == 7:
        progs[:, 3, :, 1] = [0.15, 0.05]
    rho = np.zeros((n, n), complex)
    rho[1, 1], rho[0, 0] = 0.75, 0.25
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    out = plan.simulate(flat, progs, 0.0, dt, T, F)
    if rot:
        # the rotating integrator in the lab basis, step by step
        ref = np.stack([_rotating_reference(c["generators"], flat[b], progs[b], K, dt, T, F)
                        for b in range(B)])
    else:
        _, ref = oracle.simulate(c["generators"], np.stack([rho]*B), 0.0, T*dt + 1e-14, dt, progs,
                                 K=K, W=W, nodes=nodes, F=F, vectorisation_map=vm, mode="vector",
                                 degree=20, flat_out=True)
    # the eigenbasis costs its condition number (below 100) in rounding
    assert np.abs(out - ref).max() <= (1e-11 if rot else 1e-12)


def _rotating_reference(gens, x, prog, K, dt, T, F):
    from scipy.linalg import expm
    from superspinsim_gb300.program import array_value
    W, nodes = quadrature(K)
    h = dt/F
    L0 = gens[0]
    Gk = [[expm(-L0*c*h) @ g @ expm(L0*c*h) for g in gens[1:]] for c in nodes]
    tail = expm(L0*h)
    out = np.empty((T, x.size))
    for t in range(T):
        for r in range(F):
            for e in reversed(range(K)):
                om = np.zeros_like(L0)
                for k, c in enumerate(nodes):
                    tn = ((0.0 + (r*dt)/F) + dt*t) + (dt*c)/F
                    for g in range(4):
                        om += h*W[e, k]*array_value(prog, g, tn)*Gk[k][g]
                term = x
                for j in range(1, 15):
                    term = om @ term/j
                    x = x + term
            x = tail @ x
        out[t] = x
    return out


def test_columns_long_runs_and_tables():
    """6,000 samples of one fine step: a column covers several samples; the
    same run from sampled coefficients and in two halves."""
    from superspinsim_gb300.generate_simulator import sample_table
    from superspinsim_gb300.program import array_value
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    rng = np.random.default_rng(3)
    dt, F, T = 2e-11, 1, 6000
    plan, W, nodes = _plan(c, 2, dt, F, False, True)
    progs = _programs(1, rng, 1e-4)
    rho = np.diag([0.25, 0.75, 0.0]).astype(complex)
    flat = oracle.flatten(rho, vm, N)[None]
    out = plan.simulate(flat, progs, 0.0, dt, T, F)
    _, ref = oracle.simulate(c["generators"], rho[None], 0.0, T*dt + 1e-14, dt, progs, K=2, W=W,
                             nodes=nodes, F=F, vectorisation_map=vm, mode="vector", degree=20,
                             flat_out=True)
    assert np.abs(out - ref).max() <= 1e-12

    def sampler(t, row):
        row[0] = 1.0
        for g in range(4):
            row[1 + g] = array_value(progs[0], g, t)

    tab = sample_table(sampler, 5, 0.0, dt, T, F, nodes)
    assert np.abs(plan.simulate(flat, None, 0.0, dt, T, F, table=tab) - out).max() <= 1e-12
    half = plan.simulate(out[:, T//2 - 1], progs, dt*(T//2), dt, T - T//2, F)
    assert np.abs(half - out[:, T//2:]).max() <= 1e-12


def test_columns_leave_a_prepared_batch_alone():
    """A drop-in run between a batch's prepare and its launches changes
    neither the launches' results nor the plan's report of the batch."""
    torch = pytest.importorskip("torch")
    c = load_case("nv7_n49")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    rng = np.random.default_rng(5)
    dt, F, T, B = 1e-10, 5, 6, 3
    plan, W, nodes = _plan(c, 2, dt, F, False, True)
    progs = _programs(B, rng, 1e-4)
    rho = np.zeros((7, 7), complex)
    rho[1, 1] = 1.0
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    _, fin = plan.batch(flat, progs, 0.0, dt, T, F, want_final=True)
    d_rho, d_prog = torch.from_numpy(flat).cuda(), torch.from_numpy(progs).cuda()
    plan.batch_prepare(d_rho.data_ptr(), B, d_prog.data_ptr(), 4, 2, dt, F, stream=0)
    info = plan.batch_info()
    state = d_rho.clone()
    torch.cuda.synchronize()
    plan.batch_launch(state.data_ptr(), d_prog.data_ptr(), 0.0, 0, 3, T, stream=0)
    plan.simulate(flat, progs, 0.0, dt, 2, F)
    plan.batch_launch(state.data_ptr(), d_prog.data_ptr(), 0.0, 3, 3, T, stream=0)
    torch.cuda.synchronize()
    assert np.array_equal(state.cpu().numpy(), fin)
    after = plan.batch_info()
    for key in ("lanes", "degree", "rows", "nnz", "variant", "live_generators", "live_nnz"):
        assert after[key] == info[key]


@pytest.mark.parametrize("dt", [1e-9, 1e-7, 1e-5])
def test_large_steps_keep_the_dense_exponential(dt):
    """One fine step per sample of 1 ns to 10 us (1-norms of the exponent of 20
    to 200,000) under a constant field: the matrix exponential, by sub-steps of
    the Taylor action or, beyond its range, by the dense path's scaling and
    squaring (which doubles the rounding once per squaring: 2^-53 times the
    norm)."""
    from scipy.linalg import expm
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    plan, W, nodes = _plan(c, 1, dt, 1, False, True)
    prog = np.zeros((1, 4, 1, 5))
    prog[:, :, 0, 0] = np.inf
    prog[0, 0, 0, 1] = 1e-4
    rho = np.diag([0.25, 0.75, 0.0]).astype(complex)
    flat = oracle.flatten(rho, vm, vm.shape[0])
    out = plan.simulate(flat[None], prog, 0.0, dt, 3, 1)[0]
    L = (c["generators"][0] + 1e-4*c["generators"][1])*dt
    x, E = flat, expm(L)
    for t in range(3):
        x = E @ x
        assert np.abs(out[t] - x).max() <= 1e-12 + 64*2.0**-53*np.abs(L).sum(0).max()
