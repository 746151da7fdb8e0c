"""Populations of more than 32,767 walkers in the FP64 constrained-path form: the
products of operators that keep the spins apart are two per walker in one
launch, and the launch takes every walker number that one product per walker
takes (65,535).  Against the oracle to 1e-10 per step."""
import pytest

from tests.helpers import rel_err
from tests.parity_common import STEP_TOL, compare_state, hubbard, pair_cp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decomp", ["densitySpin", "hopCharge"])
@pytest.mark.parametrize("W", [32767, 32768, 65535])
def test_step_and_measurement(decomp, W):
    m = hubbard(decomp, False, nx=2, ny=2, nup=1, ndn=1)
    g, o = pair_cp(m, W, 91, 1000, 1000)
    g.step(1)
    o.step(1)
    compare_state(g, o, STEP_TOL)
    assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
    for e in (g, o):
        e.reset_measurement()
        e.add_mixed_measurement()
    assert rel_err(g.measurement()[:2], o.measurement()[:2]) < STEP_TOL
