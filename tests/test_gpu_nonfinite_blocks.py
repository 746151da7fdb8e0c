"""A walker that is NaN throughout, in every kernel of the LU: blocked (16, 40 and
100 columns), element-wise (30 columns, many walkers), one thread block per
walker (70 and 66) and in device memory (130, and 121 and 3).  A column of NaN
has a pivot row like any other: nothing outside the walker's own matrix is read
or written.  The others match the oracle, and the status says non-finite."""
import numpy as np
import pytest

from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, molecule, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,W", [(16, 0, 4), (40, 0, 4), (100, 0, 4), (30, 0, 890), (70, 66, 4), (130, 0, 4), (121, 3, 4)])
def test_nan_walkers(nup, ndn, W):
    n = nup + 4
    g, o = pair_pl(molecule(n=n, nup=nup, ndn=ndn, G=3), W, 64, 1000, 1000, noise=0.3 / n)
    wf, lw, al = o.get_walkers()
    wf[:, :, [1, W - 1]] = np.nan
    well = [0, 2]
    o.set_walkers(wf, lw, al)
    g.set_walkers(wf, lw, al)
    lg = g.log_overlaps()
    assert not np.isfinite(lg[[1, W - 1]]).any()
    assert logov_close(lg[well], o.log_overlaps()[well], STEP_TOL) < STEP_TOL
    assert rel_err(g.green(2), o.green(2)) < STEP_TOL
    g.step(1)
    assert g.status() & 2
    al[[1, W - 1]] = 0
    for e in (g, o):
        e.set_walkers(wf, lw, al)
    assert logov_close(g.log_overlaps()[well], o.log_overlaps()[well], STEP_TOL) < STEP_TOL
    assert rel_err(g.green(0), o.green(0)) < STEP_TOL
