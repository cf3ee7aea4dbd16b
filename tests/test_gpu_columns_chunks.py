"""Drop-in runs whose propagators take several launches (2 GiB of them each): one
trajectory cut into chunks of samples, whose chain goes on across them, and
several trajectories a few at a time.  Lab frame (states written by the chain)
and rotating frame (through the eigenbasis).  The same runs in parts of one
launch each give the reference.  Tolerance: 120,000 propagators of norm below
0.1, each rounded once (2^-53 of its norm per entry and row), all in one
direction: 3e-12; in the rotating frame times the eigenbasis' condition number,
which the other runs' bound of 1e-11 for 70 samples covers ten times over."""
import numpy as np
import pytest

from conftest import load_case
from oracle import oracle
from test_gpu_columns import _plan, _programs

pytestmark = pytest.mark.gpu


def _setup(rot, B, dt, F):
    c = load_case("nv7_n49")
    plan, W, nodes = _plan(c, 2, dt, F, rot, True)
    rng = np.random.default_rng(2)
    progs = _programs(B, rng, 1e-4)
    progs[:, :, 0, 0] = 7.3e-8
    progs[:, 1] = progs[:, 0]
    progs[:, 1, :, 3] *= 1.01
    progs[:, 3, :, 1] = 0.15
    m = rng.standard_normal((7, 7)) + 1j*rng.standard_normal((7, 7))
    rho = m @ m.conj().T     # every one of the 49 rows
    rho /= np.trace(rho).real
    vm = c["vectorisation_map"]
    return plan, progs, np.stack([oracle.flatten(rho, vm, vm.shape[0])]*B)


@pytest.mark.parametrize("rot", [False, True])
def test_samples_in_several_launches(rot):
    dt, F, T = 5e-12, 1, 120000     # 111,848 samples fill 2 GiB
    plan, progs, flat = _setup(rot, 1, dt, F)
    out = plan.simulate(flat, progs, 0.0, dt, T, F)
    tol = 1e-10 if rot else 3e-12
    x, at = flat, 0
    for n in (50000, 50000, 20000):
        part = plan.simulate(x, progs, dt*at, dt, n, F)
        assert np.abs(out[:, at:at + n] - part).max() <= tol
        x, at = part[:, -1], at + n


def test_trajectories_in_several_launches():
    dt, F, T, B = 5e-12, 1, 50000, 3
    plan, progs, flat = _setup(False, B, dt, F)
    out = plan.simulate(flat, progs, 0.0, dt, T, F)
    for b in range(B):
        one = plan.simulate(flat[b:b + 1], progs[b:b + 1], 0.0, dt, T, F)
        assert np.abs(out[b] - one[0]).max() <= 3e-12
