"""Drop-in programs with an infinite offset, amplitude, frequency or phase are
refused (the state becomes NaN) also on a channel whose generator moves no row
that is reachable from the initial state."""
import numpy as np
import pytest

from conftest import load_case, quadrature
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [1, 2, 3, 4])
@pytest.mark.parametrize("channel", [0, 2])
def test_infinite_coefficient_is_refused(channel, field):
    from superspinsim_gb300 import _lib
    c = load_case("spin1_c1")
    vm = c["vectorisation_map"]
    W, nodes = quadrature(2)
    plan = _lib.Plan(c["generators"], W, nodes)
    rho = np.diag([0.25, 0.75, 0.0]).astype(complex)   # the z field moves no population
    flat = oracle.flatten(rho, vm, vm.shape[0])[None]
    prog = np.zeros((1, 4, 1, 5))
    prog[:, :, 0, 0] = np.inf
    prog[0, channel, 0, 1:] = (1e-5, 1e-4, 1e9, 0.3)
    assert np.isfinite(plan.simulate(flat, prog, 0.0, 1e-10, 3, 5)).all()
    for v in (np.inf, -np.inf):
        prog[0, channel, 0, field] = v
        with pytest.raises(_lib.SSSError) as e:
            plan.simulate(flat, prog, 0.0, 1e-10, 3, 5)
        assert "ENONFINITE" in str(e.value)
