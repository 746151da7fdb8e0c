"""The blocked LU at the edges of its panels, warps and column halves, against
the oracle (plain FP64 form, 1e-10).

Panels are 8 columns wide, a CTA holds 64 columns and a cluster of two CTAs up
to 128; two spin blocks of up to 64 columns share a cluster.  Log-overlaps,
Green's functions (the inverse), population-control weights and tables (the
elimination without the inverse) are compared; walkers equal to the trial give
the identity with its ties and zeros.
"""
import pytest

from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, compare_state, molecule, pair_pl

pytestmark = pytest.mark.gpu


def check(n, nup, ndn, W, noise):
    m = molecule(n=n, nup=nup, ndn=ndn, G=4)
    seed = 500 + nup
    g, o = pair_pl(m, W, seed, 1000, 1000, noise=noise)
    assert logov_close(g.log_overlaps(), o.log_overlaps(), STEP_TOL) < STEP_TOL
    for spin in range(2 if ndn else 1):
        assert rel_err(g.green(W - 1, spin), o.green(W - 1, spin)) < STEP_TOL
    tg, wg = g.pop_control()
    to, wo = o.pop_control()
    assert rel_err(wg, wo) < STEP_TOL
    assert (tg == to).all()
    compare_state(g, o, STEP_TOL)


@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 15, 16, 17, 32, 33, 40, 63, 64, 65, 72, 73, 96, 119, 120, 121, 127, 128])
def test_one_block(N):
    check(N + 3, N, 0, 3, 0.3 / (N + 3) ** 0.5)


@pytest.mark.parametrize("nup,ndn", [(1, 1), (8, 3), (16, 16), (33, 1), (40, 33), (64, 17), (64, 64)])
def test_two_blocks(nup, ndn):
    check(nup + 5, nup, ndn, 3, 0.3 / (nup + 5) ** 0.5)


@pytest.mark.parametrize("N", [5, 16, 50, 70])
def test_walkers_equal_to_the_trial(N):
    check(N + 4, N, 0, 2, 0.0)


def test_many_walkers_of_17_to_32_columns():
    """Both sides of the rule that leaves 25 to 32 columns to the element-wise kernel."""
    for N, W in ((24, 900), (25, 888), (25, 889)):
        check(30, N, 0, W, 0.05)
