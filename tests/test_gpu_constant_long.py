"""Constant samples of long programs: forty segments whose ends are out of order,
repeated, infinite or past, mostly constant (every kernel that knows the maps
takes them) and mostly varying (groups that share a warp step all samples), in
one-shot runs and in chunks.  Against the oracle."""
import numpy as np
import pytest

from test_gpu_constant import _reference, _setup

pytestmark = pytest.mark.gpu


def _programs(B, S, dt, T, rng, varying):
    p = np.zeros((B, 4, S, 5))
    p[..., 0] = -np.inf
    for b in range(B):
        for ch, s_used in ((0, S), (3, S//2)):
            ends = np.sort(rng.uniform(0, T*dt, s_used))
            ends[rng.integers(0, s_used, s_used//4)] = rng.choice([-1.0, 0.0, 2*dt, 5*dt, -np.inf], s_used//4)
            if b % 3 == 1:
                k = rng.permutation(s_used)[:6]
                ends[k] = ends[k[::-1]]
            if b % 3 == 2:
                ends[-1] = np.inf
            p[b, ch, :s_used, 0] = ends
        on = rng.random(S) < (0.9 if varying else 0.2)
        p[b, 0, on, 2] = 1e-4*rng.uniform(0.5, 1, on.sum())
        p[b, 0, :, 3] = 3.1e9
        p[b, 3, :S//2, 1] = rng.choice([0.0, 0.15], S//2)
    return p


@pytest.mark.parametrize("varying", [False, True])
@pytest.mark.parametrize("variant,lanes", [(0, 0), (6, 8), (6, 128), (7, 32), (8, 32), (8, 128)])
def test_long_programs_against_oracle(variant, lanes, varying):
    torch = pytest.importorskip("torch")
    from superspinsim_gb300 import _lib
    dt, T, F, B, S = 1e-10, 60, 8, 9, 40
    c, vm, N, _, rho, W, nodes, _, flat = _setup(0, 0, B=B)
    progs = _programs(B, S, dt, T, np.random.default_rng(21), varying)
    plan = _lib.Plan(c["generators"], W, nodes)
    plan.set_batch_config(lanes=lanes, variant=variant)
    try:
        _, fin, tr = plan.batch(flat, progs, 0.0, dt, T, F, want_final=True, want_trace=True)
    except _lib.SSSError as e:
        # two varying coefficients outgrow 32 lanes
        assert (variant, lanes) == (8, 32) and "no layout fits" in str(e)
        return
    ref = _reference(c, vm, progs, rho, W, nodes, 0.0, dt, T, F)
    assert np.abs(tr - ref).max() <= 1e-12
    d_prog, state = torch.from_numpy(progs).cuda(), torch.from_numpy(flat).cuda()
    plan.batch_prepare(state.data_ptr(), B, d_prog.data_ptr(), 4, S, dt, F, stream=0)
    torch.cuda.synchronize()
    for t in range(0, T, 7):
        plan.batch_launch(state.data_ptr(), d_prog.data_ptr(), 0.0, t, min(7, T - t), T, stream=0)
    torch.cuda.synchronize()
    assert np.array_equal(state.cpu().numpy(), fin)
