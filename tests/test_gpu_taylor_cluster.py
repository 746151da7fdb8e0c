"""The FP64 Taylor kernel over its cluster sizes, two to eight blocks of 16
columns per walker: the stopping test meets across the cluster.  Dead walkers
leave as whole clusters.  Against the oracle to the FP64 form's 1e-10 per step."""
import pytest

from tests.helpers import rel_err
from tests.parity_common import STEP_TOL, compare_state, molecule, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N", [(33, 32), (50, 48), (66, 64), (80, 65), (100, 96), (112, 112), (130, 128)])
def test_step(n, N):
    g, o = pair_pl(molecule(n=n, nup=N, ndn=0, G=4), 3, 23, 1000, 1000, noise=0.3 / n)
    for _ in range(2):
        wf, lw, al = o.get_walkers()
        al[1] = 0
        o.set_walkers(wf, lw, al)
        g.set_walkers(wf, lw, al)
        g.set_rng(23, o.rng_counter())
        g.step(1)
        o.step(1)
        compare_state(g, o, STEP_TOL)
        assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
