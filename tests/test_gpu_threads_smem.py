"""Two plans on two host threads: one launches clusters that take nearly all of
an SM's shared memory, the other prepares batches of a smaller large system
(which asks how many clusters of the same kernel the GPU holds).  The kernel's
shared-memory limit belongs to the process: no launch may fail for the other
thread's query, and the results are those of the plan alone."""
import threading

import numpy as np
import pytest

from conftest import quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_prepare_beside_launches_of_large_clusters():
    torch = pytest.importorskip("torch")
    from superspinsim_gb300 import _lib, models
    from superspinsim_gb300.generators import generate_atoms
    W, nodes = quadrature(2)
    # a field off the axis: 72,000 entries, 228 KB on each of 4 CTAs
    spins, inter, groups = models.nv_21(0.05*np.array([np.sin(0.5), 0.0, np.cos(0.5)]),
                                        params=models.nv21_params())
    g, vm = generate_atoms(spins, inter, groups, use_incoherent=False)
    vm = np.asarray(vm)
    gens = np.array([g["generators"][k] for k in ("L0", "Gx", "Gy", "Gz", "Gr")])
    N, B, T, F, dt = vm.shape[0], 20, 400, 1, 1e-11
    rho = np.zeros((21, 21), complex)
    for k in range(3, 6):
        rho[k, k] = 1/3
    flat = np.stack([oracle.flatten(rho, vm, N)]*B)
    progs = np.zeros((B, 4, 1, 5))
    progs[:, :, 0, 0] = np.inf
    progs[:, 0, 0, 2] = 1.78e-4
    progs[:, 0, 0, 3] = 4.27e9
    progs[:, 3, 0, 1] = 0.15
    big = _lib.Plan(gens, W, nodes)
    big.set_batch_config(variant=8)
    d_prog, state = torch.from_numpy(progs).cuda(), torch.from_numpy(flat).cuda()
    big.batch_prepare(state.data_ptr(), B, d_prog.data_ptr(), 4, 1, dt, F, stream=0)
    assert big.batch_info()["variant"] == 8

    # a chain of 70 levels: one more row than the one-CTA kernels hold, and some
    n = 70
    L = np.zeros((5, n, n))
    L[0] = 1e9*(np.eye(n, k=-1) - np.eye(n))
    L[1] = 1e12*(np.eye(n, k=-1) - np.eye(n, k=1))
    small = _lib.Plan(L, W, nodes)
    small.set_batch_config(variant=8)
    x = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    x[:, 0] = 1.0
    p3 = torch.from_numpy(progs[:3].copy()).cuda()
    torch.cuda.synchronize()
    errors, stop = [], threading.Event()

    def prepares():
        try:
            while not stop.is_set():
                small.batch_prepare(x.data_ptr(), 3, p3.data_ptr(), 4, 1, dt, F, stream=0)
        except Exception as e:   # reported by the test below
            errors.append(e)

    other = threading.Thread(target=prepares)
    other.start()
    try:
        for t in list(range(T))*30:
            big.batch_launch(state.data_ptr(), d_prog.data_ptr(), 0.0, t, 1, T, stream=0)
    finally:
        stop.set()
        other.join()
    torch.cuda.synchronize()
    assert not errors
    assert small.batch_info()["variant"] == 8
    alone = torch.from_numpy(flat).cuda()
    for _ in range(30):
        big.batch_launch(alone.data_ptr(), d_prog.data_ptr(), 0.0, 0, T, T, stream=0)
    torch.cuda.synchronize()
    assert torch.equal(alone, state)
