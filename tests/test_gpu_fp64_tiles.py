"""FP64 products at the edges of their tiles, against the oracle.

The FP64 GEMM works in 8-row granules, 32- and 64-row tiles and 8- or
16-column stages; the Taylor kernel holds 16 rows per warp and 16 columns per
CTA, one cluster per walker, up to n = 256.  Sizes sit on either side of
those boundaries (n = 257 runs the series order by order).  Per step the
engine and the oracle must agree to the FP64 form's criterion, 1e-10.
"""
import pytest

from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, compare_state, molecule, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nup,ndn,G,W", [(5, 2, 1, 3, 1), (8, 8, 0, 7, 3), (15, 4, 4, 9, 5), (17, 9, 8, 33, 2),
                                           (31, 16, 15, 40, 3), (63, 17, 16, 65, 3), (65, 33, 32, 64, 2),
                                           (129, 49, 7, 31, 2), (255, 5, 3, 9, 2), (257, 18, 2, 6, 2)])
def test_step_and_measurement_at_tile_edges(n, nup, ndn, G, W):
    m = molecule(n=n, nup=nup, ndn=ndn, G=G)
    seed = 400 + n
    g, o = pair_pl(m, W, seed, 1000, 1000, noise=0.02)
    for _ in range(2):
        wf, lw, al = o.get_walkers()
        g.set_walkers(wf, lw, al)
        g.set_rng(seed, o.rng_counter())
        g.step(1)
        o.step(1)
        compare_state(g, o, STEP_TOL)
        assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
    wf, lw, al = o.get_walkers()
    g.set_walkers(wf, lw, al)
    for e in (g, o):
        e.reset_measurement()
        e.add_mixed_measurement()
    assert rel_err(g.measurement()[:3], o.measurement()[:3]) < STEP_TOL
    for a, b in zip(g.cholesky_nums(), o.cholesky_nums()):
        assert rel_err(a, b) < STEP_TOL
    assert logov_close(g.log_overlaps(), o.log_overlaps(), STEP_TOL) < STEP_TOL
