"""Contractions cut into pieces: the force and the exchange's quadratic forms
of few output tiles are partial products over K = electrons x orbitals, in
pieces that divide neither K nor the row blocks, end before a row block's
diagonal, or leave a row block empty.  Against the oracle to the FP64 form's
1e-10; small K (one piece), K around multiples of the 64-element granule, one
walker and one vector."""
import pytest

from tests.helpers import rel_err
from tests.parity_common import STEP_TOL, molecule, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nup,ndn,G,W", [(4, 1, 1, 2, 1), (13, 5, 4, 1, 3), (21, 9, 3, 40, 1), (32, 10, 8, 33, 35),
                                           (37, 11, 11, 20, 70), (43, 12, 9, 65, 33), (48, 16, 4, 36, 6)])
def test_force_and_exchange(n, nup, ndn, G, W):
    m = molecule(n=n, nup=nup, ndn=ndn, G=G)
    g, o = pair_pl(m, W, 31, 1000, 1000, noise=0.02)
    for e in (g, o):
        e.reset_measurement()
        e.add_mixed_measurement()
    assert rel_err(g.measurement()[:3], o.measurement()[:3]) < STEP_TOL
    for a, b in zip(g.cholesky_nums(), o.cholesky_nums()):
        assert rel_err(a, b) < STEP_TOL
    g.step(1)
    o.step(1)
    assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
