"""Which group widths hold the power series of which system: 1 to 19 reachable
rows, none, one and two varying coefficients.  A packing that stops fitting fails
here (the comparison with the oracle takes a width that holds none as nothing to
compare)."""
import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu

FITS = {("qubit_couple_res_e2", 2, 1): (16, 32, 64, 128), ("spin1_c1", 1, 1): (16, 32, 64, 128),
        ("spin1_c1", 2, 0): (16, 32, 64, 128), ("spin1_c1", 2, 2): (64, 128),
        ("spin1_c1", 5, 1): (16, 32, 64, 128), ("nv7_n19", 2, 1): (32, 64, 128),
        ("nv7_n49", 2, 2): (128,)}


@pytest.mark.parametrize("lanes", [16, 32, 64, 128])
@pytest.mark.parametrize("name,K,drives", list(FITS))
def test_widths_that_hold_a_layout(name, K, drives, lanes):
    from superspinsim_gb300 import _lib
    c = load_case(name)
    vm = c["vectorisation_map"]
    N = vm.shape[0]
    n = int(vm[:, 0].max()) + 1
    progs = np.zeros((1, 4, 1, 5))
    progs[..., 0] = np.inf
    progs[0, :drives, 0, 1:3] = (1e-5, 1e-4)
    progs[0, :drives, 0, 3] = 28e6 if name.startswith("qubit") else 3.15e9
    if n == 7:
        progs[0, 3, 0, 1] = 0.15
    rho = np.zeros((n, n), complex)
    rho[1, 1], rho[0, 0] = 0.75, 0.25
    W, nodes = quadrature(K)
    plan = _lib.Plan(c["generators"], W, nodes)
    plan.set_batch_config(lanes=lanes, variant=8)
    flat = oracle.flatten(rho, vm, N)[None]
    try:
        plan.batch(flat, progs, 0.0, 1e-10, 1, 21, want_final=True)
        fits = True
    except _lib.SSSError as e:
        assert "no layout fits" in str(e)
        fits = False
    assert fits == (lanes in FITS[name, K, drives])
