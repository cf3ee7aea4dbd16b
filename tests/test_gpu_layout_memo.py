"""A plan remembers the layouts of its last sixteen batch shapes: with sixteen of
them known, a call with one of them is still fast (no new search), and the
results of the remembered layout are those of a new plan."""
import time

import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


def test_full_memo_keeps_what_it_knows():
    from superspinsim_gb300 import _lib
    c = load_case("nv7_n49")
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    W, nodes = quadrature(2)
    rho = np.zeros((7, 7), complex)
    rho[1, 1] = 1.0
    flat = oracle.flatten(rho, vm, N)[None]
    progs = np.zeros((1, 4, 1, 5))
    progs[..., 0] = np.inf
    progs[0, :3, 0, 2:4] = (1e-4, 3.1e9)   # three drives: no power series

    def call(plan, threads, laser):
        plan.set_batch_config(cta_threads=threads)
        progs[0, 3, 0, 1:4] = (0.1, 0.05, 1e7) if laser else 0.0
        t = time.perf_counter()
        _, fin = plan.batch(flat, progs, 0.0, 1e-10, 1, 4, want_final=True)
        return time.perf_counter() - t, fin

    plan = _lib.Plan(c["generators"], W, nodes)
    shapes = [(32*k, laser) for laser in (False, True) for k in range(1, 9)]
    search = [call(plan, *s) for s in shapes]
    known, fin = call(plan, *shapes[-2])
    # a search over the lane counts takes milliseconds
    assert known < 0.3*min(t for t, _ in search)
    assert np.array_equal(fin, search[-2][1])
    assert np.array_equal(fin, call(_lib.Plan(c["generators"], W, nodes), *shapes[-2])[1])
