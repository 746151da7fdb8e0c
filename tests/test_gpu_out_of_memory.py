"""An allocation that fails is the failing call's error and nobody else's: the
next engine is made, and runs, as if it had not been."""
import pytest

from afqmclab_b200 import capi
from tests.parity_common import STEP_TOL, compare_state, hubbard, molecule, pair_cp, pair_pl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("late", [False, True])
def test_engines_after_a_failed_one(late):
    for make, pair, m in ((capi.cp_engine, pair_cp, hubbard()), (capi.pl_engine, pair_pl, molecule())):
        with pytest.raises(capi.AfqmcError, match="out of memory"):
            if late:   # the exchange's square matrices of 150,000 rows
                capi.pl_engine(molecule(n=600, nup=250, ndn=0, G=1), 2, 5, 10, 10)
            else:      # terabytes of walkers
                make(m, 2_000_000_000, 5, 10, 10)
        g, o = pair(m, 4, 94, 1000, 1000)
        g.step(1)
        o.step(1)
        compare_state(g, o, STEP_TOL)
