"""Output samples over which nothing varies, taken by one map (sss_constant.h),
against the oracle: pulse protocols whose segments end on and inside samples,
every kernel that knows the maps, trajectories that start past zero, and
programs whose constant values changed after the batch was prepared."""
import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


def _pulses(B, rng, two_levels):
    """Laser / pulse / dark / pulse / laser; some ends fall inside samples."""
    inf = np.inf
    p = np.zeros((B, 4, 5, 5))
    p[:, :, :, 0] = -inf
    for b in range(B):
        e = np.cumsum([3e-10, 2e-10, 6e-10, 2e-10]) + (0.0 if b % 2 else 3.7e-11)
        f = 3.15e9*rng.uniform(0.9, 1.1)
        for s, amp in enumerate((0.0, 1e-4, 0.0, 2e-4, 0.0)):
            p[b, 0, s] = (e[s] if s < 4 else inf, 0, amp, f, 0.3*b)
        lvl = 0.2 if two_levels and b % 3 == 0 else 0.15
        p[b, 3, 0] = (e[0], lvl, 0, 0, 0)
        p[b, 3, 1] = (e[3], 0, 0, 0, 0)
        p[b, 3, 2] = (inf, lvl, 0, 0, 0)
    return p


def _setup(variant, lanes, two_levels=False, B=7):
    from superspinsim_gb300 import _lib
    c = load_case("nv7_n19")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    rng = np.random.default_rng(8)
    progs = _pulses(B, rng, two_levels)
    rho = np.zeros((7, 7), complex)
    rho[1, 1], rho[0, 0] = 0.75, 0.25
    W, nodes = quadrature(2)
    plan = _lib.Plan(c["generators"], W, nodes)
    plan.set_batch_config(lanes=lanes, variant=variant)
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    return c, vm, N, progs, rho, W, nodes, plan, flat


def _reference(c, vm, progs, rho, W, nodes, t0, dt, T, F):
    _, ref = oracle.simulate(c["generators"], np.stack([rho]*len(progs)), t0, t0 + T*dt + 1e-14, dt,
                             progs, K=2, W=W, nodes=nodes, F=F, vectorisation_map=vm, mode="vector",
                             degree=20, flat_out=True)
    return ref


@pytest.mark.parametrize("variant,lanes", [(0, 0), (6, 16), (6, 128), (7, 32), (8, 128)])
@pytest.mark.parametrize("F,t0,two_levels", [(8, 0.0, False), (9, 1.3e-10, True)])
def test_constant_samples_against_oracle(variant, lanes, F, t0, two_levels):
    dt, T = 1e-10, 16
    c, vm, N, progs, rho, W, nodes, plan, flat = _setup(variant, lanes, two_levels)
    samples = np.array([T, T - 1, 5, 0, 1, T, 9], dtype=np.int32)
    w = np.random.default_rng(1).uniform(-1, 1, N)
    ro, fin, tr = plan.batch(flat, progs, t0, dt, T, F, samples=samples, readout_weights=w,
                             want_final=True, want_trace=True)
    ref = _reference(c, vm, progs, rho, W, nodes, t0, dt, T, F)
    for b, s in enumerate(samples):
        last = ref[b, s - 1] if s else flat[b]
        assert np.abs(fin[b] - last).max() <= 1e-12
        assert np.abs(tr[b, :s] - ref[b, :s]).max(initial=0.0) <= 1e-12
        assert np.abs(ro[b, :s] - ref[b, :s] @ w).max(initial=0.0) <= 1e-12


def test_values_changed_after_prepare():
    """A prepared batch whose programs get other constant values (no larger)
    steps them: the maps belong to the values they were made for."""
    torch = pytest.importorskip("torch")
    dt, T, F = 1e-10, 16, 8
    c, vm, N, progs, rho, W, nodes, plan, flat = _setup(0, 0)
    B = len(progs)
    d_rho, d_prog = torch.from_numpy(flat).cuda(), torch.from_numpy(progs).cuda()
    plan.batch_prepare(d_rho.data_ptr(), B, d_prog.data_ptr(), 4, 5, dt, F, stream=0)
    changed = progs.copy()
    changed[:, 3, :, 1] *= 0.5
    changed[1, 3, 2, 1] = 0.15
    d_prog.copy_(torch.from_numpy(changed))
    state = d_rho.clone()
    torch.cuda.synchronize()
    plan.batch_launch(state.data_ptr(), d_prog.data_ptr(), 0.0, 0, T, T, stream=0)
    torch.cuda.synchronize()
    ref = _reference(c, vm, changed, rho, W, nodes, 0.0, dt, T, F)
    assert np.abs(state.cpu().numpy() - ref[:, -1]).max() <= 1e-12
