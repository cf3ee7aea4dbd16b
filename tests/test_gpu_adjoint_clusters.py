"""Gradients whose forward pass runs on clusters (21-level NV, the drive alone
varying under a constant laser): the states that k_power_big stores, in its own
row order, give the row-part kernels' objective and gradients, for clusters of 8,
4 and 2 CTAs and in chunks of stored states.  Tolerance: 160 exponentials forward
and back, each rounding a row of at most 128 products and sums: 5e-12 of the
largest entry."""
import numpy as np
import pytest

from conftest import load_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,chunked", [(2, False), (20, False), (20, True), (60, False)])
def test_forward_on_clusters(B, chunked):
    from superspinsim_gb300.adjoint import Objective, trapezoid_weights
    c = load_case("nv21_n441")
    rho = np.zeros((21, 21), complex)
    for k in range(3, 6):
        rho[k, k] = 1/3
    dt, T, F, S = 2e-10, 4, 20, 3
    obj = Objective(c["generators"], c["vectorisation_map"], rho, list(range(9, 18)), 65.9e6,
                    number_of_fine_divisions=F)
    rng = np.random.default_rng(B)
    progs = np.zeros((B, 4, S, 5))
    progs[:, :, :, 0] = [2.5e-10, 5.1e-10, np.inf]
    progs[:, 0, :, 2] = 5e-4*rng.uniform(0.3, 1, (B, S))
    progs[:, 0, :, 3] = 4.27e9
    progs[:, 0, :, 4] = rng.uniform(0, 6, (B, S))
    progs[:, 3, :, 1] = 0.15
    tw = trapezoid_weights(T, dt, 0, T - 1)
    out = {}
    for variant in (4, 0):
        obj.plan.set_batch_config(variant=variant)
        if variant == 0 and chunked:
            obj.plan.set_adjoint_memory(7*T*F*2*obj.plan.batch_info()["rows"]*8 + 8)
        out[variant] = obj.run(progs, dt, T, tw) + obj.run(progs, dt, T, tw, channel=0)
        if variant == 0:
            assert obj.plan.last_launches() == (2*3 if chunked else 2)
    for a, b in zip(out[0], out[4]):
        assert np.abs(a - b).max() <= 5e-12*np.abs(b).max()
    # another forward kernel ran: the same sums in another order
    assert not np.array_equal(out[0][0], out[4][0])
