"""The adjoint's scratch is the engine's and is reused: repeated evaluations,
with and without the Cholesky gradient, from other walkers in between, give
the same numbers to the last bit as a fresh engine does."""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs
from tests.parity_common import molecule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn", [(5, 5), (5, 3)])
def test_repeated_evaluations(nup, ndn):
    m = molecule(n=12, nup=nup, ndn=ndn, G=7)
    W = 19
    pops = [inputs.initial_walkers(m.phiTUp, W, seed=s, noise=0.05) for s in (1, 2)]

    def evaluate(e, k, chol):
        e.set_walkers(*pops[k])
        r = e.adjoint(want_chol=chol)
        return [r["E"], r["mean_logov"], r["dE_dt"], *r["dE_dconj_phiT"], *r["dlogov_dconj_phiT"]] + ([r["dE_dchol"]] if chol else [])

    e = capi.pl_engine(m, W, 3)
    for k, chol in ((0, True), (1, False), (1, True), (0, False), (0, True)):
        f = capi.pl_engine(m, W, 3)
        for a, b in zip(evaluate(e, k, chol), evaluate(f, k, chol)):
            assert np.array_equal(a, b)
        f.close()
    e.close()
