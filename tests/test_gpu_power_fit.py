"""Sweeps of the 21-level NV whose power series outgrows the shared memory of
the cluster that would keep every trajectory resident: they take a larger
cluster in turns, or the Taylor kernels, and match the oracle."""
import math

import numpy as np
import pytest

from conftest import quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tilt,F,amp,B", [(0.5, 100, 2.14e-4, 20), (0.5, 100, 2.14e-4, 36),
                                          (0.0, 33, 5.35e-4, 60), (0.0, 100, 1.8e-4, 100)])
def test_series_beyond_the_resident_cluster(tilt, F, amp, B):
    from superspinsim_gb300 import _lib, models
    from superspinsim_gb300.generators import generate_atoms
    field = 0.05*np.array([math.sin(tilt), 0.0, math.cos(tilt)])
    spins, inter, groups = models.nv_21(field, params=models.nv21_params())
    g, vm = generate_atoms(spins, inter, groups, use_incoherent=False)
    vm = np.asarray(vm)
    gens = np.array([g["generators"][k] for k in ("L0", "Gx", "Gy", "Gz", "Gr")])
    N = vm.shape[0]
    rho = np.zeros((21, 21), complex)
    for k in range(3, 6):
        rho[k, k] = 1/3
    rng = np.random.default_rng(B)
    dt = 1e-9
    progs = np.zeros((B, 4, 1, 5))
    progs[:, :, 0, 0] = np.inf
    progs[:, 0, 0, 2] = amp
    progs[:, 0, 0, 3] = 4.27e9 + rng.uniform(-3e7, 3e7, B)
    progs[:, 3, 0, 1] = 10/65.9
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    W, nodes = quadrature(2)
    plan = _lib.Plan(gens, W, nodes)
    _, fin = plan.batch(flat, progs, 0.0, dt, 1, F, want_final=True)
    for b in sorted({0, B//2, B - 1}):
        _, ref = oracle.simulate(gens, rho[None], 0.0, dt + 1e-14, dt, progs[b:b + 1], K=2, W=W,
                                 nodes=nodes, F=F, vectorisation_map=vm, mode="vector", degree=20,
                                 flat_out=True)
        assert np.abs(fin[b] - ref[0, 0]).max() <= 1e-12
