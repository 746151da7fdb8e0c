"""Columns per CTA in the FP64 Taylor kernel: walkers of 17 to 24 columns in one
CTA (n <= 96; small matrices only above 148 walkers), a cluster of 16-column
CTAs next to them.  Against the oracle to the FP64 form's 1e-10 per step."""
import pytest

from tests.helpers import rel_err
from tests.parity_common import STEP_TOL, compare_state, molecule, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nup,ndn,W", [(24, 17, 9, 149), (40, 24, 24, 149), (40, 24, 3, 148), (41, 24, 17, 2),
                                         (41, 25, 8, 2), (81, 21, 14, 2), (96, 24, 20, 2), (97, 20, 20, 2), (64, 16, 16, 3)])
def test_step(n, nup, ndn, W):
    g, o = pair_pl(molecule(n=n, nup=nup, ndn=ndn, G=6), W, 19, 1000, 1000, noise=0.02)
    for _ in range(2):
        wf, lw, al = o.get_walkers()
        g.set_walkers(wf, lw, al)
        g.set_rng(19, o.rng_counter())
        g.step(1)
        o.step(1)
        compare_state(g, o, STEP_TOL)
        assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
