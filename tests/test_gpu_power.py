"""The power-series batched kernels (variant 8) against the oracle: every
group width, one to nineteen reachable rows, none, one and two varying
coefficients, one table (CF2:1, CF4:2) and several (CF6:5), uneven lengths
and trajectories that outlast the coefficient ring."""
import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [0, 16, 32, 64, 128])
@pytest.mark.parametrize("name,K,drives", [("qubit_couple_res_e2", 2, 1), ("spin1_c1", 1, 1),
                                           ("spin1_c1", 2, 0), ("spin1_c1", 2, 2),
                                           ("spin1_c1", 5, 1), ("nv7_n19", 2, 1),
                                           ("nv7_n49", 2, 2)])
def test_power_series_against_oracle(name, K, drives, lanes):
    from superspinsim_gb300 import _lib
    c = load_case(name)
    vm = c["vectorisation_map"]
    gens = c["generators"]
    N = vm.shape[0]
    n = int(vm[:, 0].max()) + 1
    rng = np.random.default_rng(17)
    B, T, F, dt = 5, 5, 21, 1e-10
    f0 = 28e6 if name.startswith("qubit") else 3.15e9
    progs = np.zeros((B, 4, 2, 5))
    progs[:, :, 0, 0] = 2.3e-10
    progs[:, :, 1, 0] = np.inf
    for ch in range(drives):
        progs[:, ch, :, 1] = 1e-5*rng.uniform(-1, 1, (B, 2))
        progs[:, ch, :, 2] = 1e-4*rng.uniform(0.2, 1, (B, 2))
        progs[:, ch, :, 3] = f0*rng.uniform(0.9, 1.1, (B, 2))
        progs[:, ch, :, 4] = rng.uniform(0, 6, (B, 2))
    if n == 7:
        progs[:, 3, :, 1] = 0.15
    samples = np.array([T, 0, 1, T - 1, T], dtype=np.int32)
    rho = np.zeros((n, n), complex)
    rho[1, 1], rho[0, 0] = 0.75, 0.25
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    w = rng.uniform(-1, 1, N)
    W, nodes = quadrature(K)
    plan = _lib.Plan(gens, W, nodes)
    plan.set_batch_config(lanes=lanes, variant=8)
    try:
        ro, fin, tr = plan.batch(flat, progs, 0.0, dt, T, F, samples=samples, readout_weights=w,
                                 want_final=True, want_trace=True)
    except _lib.SSSError as e:
        # more entries than this width's largest program holds
        assert e.code == -1 and "no layout fits" in str(e)
        assert lanes in (16, 32) or (n == 7 and drives == 2)
        return
    assert plan.batch_info()["variant"] == 8
    _, ref = oracle.simulate(gens, np.stack([rho]*B), 0.0, T*dt + 1e-14, dt, progs, K=K, W=W,
                             nodes=nodes, F=F, vectorisation_map=vm, mode="vector", degree=20,
                             flat_out=True)
    for b, s in enumerate(samples):
        last = ref[b, s - 1] if s else flat[b]
        assert np.abs(fin[b] - last).max() <= 1e-12
        assert np.abs(tr[b, :s] - ref[b, :s]).max(initial=0.0) <= 1e-12
        assert np.abs(ro[b, :s] - ref[b, :s] @ w).max(initial=0.0) <= 1e-12
        assert not tr[b, s:].any() and not ro[b, s:].any()


@pytest.mark.parametrize("B", [1, 5, 20, 40, 80, 170])
def test_large_system_clusters_against_oracle(B):
    """The 21-level NV (171 reachable rows) on clusters of 8, 4, 2 and 1 CTAs
    per trajectory: uneven lengths past the coefficient ring (64 steps; 16 for
    one CTA), readouts, traces and final states of trajectories from both ends
    of the batch."""
    from superspinsim_gb300 import _lib
    c = load_case("nv21_n441")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    rng = np.random.default_rng(B)
    T, F, dt = 2, 40, 2e-10
    progs = np.zeros((B, 4, 1, 5))
    progs[:, :, 0, 0] = np.inf
    progs[:, 0, 0, 2] = 2e-4*rng.uniform(0.5, 1, B)
    progs[:, 0, 0, 3] = 4.27e9 + rng.uniform(-3e7, 3e7, B)
    progs[:, 3, 0, 1] = 0.15
    samples = np.full(B, T, dtype=np.int32)
    samples[-1] = 1
    rho = np.zeros((21, 21), complex)
    for k in range(3, 6):
        rho[k, k] = 1/3
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    w = rng.uniform(-1, 1, N)
    W, nodes = quadrature(2)
    plan = _lib.Plan(c["generators"], W, nodes)
    plan.set_batch_config(variant=8)
    ro, fin, tr = plan.batch(flat, progs, 0.0, dt, T, F, samples=samples, readout_weights=w,
                             want_final=True, want_trace=True)
    assert plan.batch_info()["variant"] == 8
    for b in sorted({0, B//2, B - 1}):
        _, ref = oracle.simulate(c["generators"], rho[None], 0.0, T*dt + 1e-14, dt, progs[b:b + 1],
                                 K=2, W=W, nodes=nodes, F=F, vectorisation_map=vm, mode="vector",
                                 degree=20, flat_out=True)
        s = samples[b]
        assert np.abs(fin[b] - ref[0, s - 1]).max() <= 1e-12
        assert np.abs(tr[b, :s] - ref[0, :s]).max() <= 1e-12
        assert np.abs(ro[b, :s] - ref[0, :s] @ w).max() <= 1e-12
        assert not tr[b, s:].any() and not ro[b, s:].any()


@pytest.mark.parametrize("name,B", [("spin1_c1", 5), ("nv7_n19", 700), ("nv21_n441", 3)])
def test_chunks_and_graph_replay(name, B):
    """Chunked launches and their CUDA graph give the one-shot run bit for bit
    on the row-aligned, the 32-lane and the cluster kernels."""
    torch = pytest.importorskip("torch")
    from superspinsim_gb300.sweep import ChunkedRun, Sweep
    c = load_case(name)
    vm = c["vectorisation_map"]
    n = int(vm[:, 0].max()) + 1
    rng = np.random.default_rng(4)
    T, F, dt = 5, 9, 1e-10
    progs = np.zeros((B, 4, 1, 5))
    progs[:, :, 0, 0] = np.inf
    progs[:, 0, 0, 2] = 1e-4*rng.uniform(0.5, 1, B)
    progs[:, 0, 0, 3] = 3.0e9 + rng.uniform(-3e7, 3e7, B)
    rho = np.zeros((n, n), complex)
    rho[1, 1] = 1.0
    w = rng.uniform(-1, 1, vm.shape[0])
    sw = Sweep(c["generators"], vm, number_of_exponentials=2, number_of_fine_divisions=F)
    one = sw.run(rho, progs, 0.0, T*dt + 1e-14, dt, readout_weights=w, final_state=True)
    assert sw.info()["variant"] == 8
    for run in (ChunkedRun(sw, rho, progs, 0.0, dt, T, readout_weights=w).run(chunk=2),
                ChunkedRun(sw, rho, progs, 0.0, dt, T, readout_weights=w).capture(chunk=3).replay()):
        torch.cuda.synchronize()
        r = run.results()
        assert np.array_equal(r["readout"], one["readout"])
        assert np.array_equal(r["final"], one["final"])
