"""The mixed form's sums per Cholesky vector do not depend on the electrons' order.

The pair matrix of the exchange has the walkers' weights rounded to bf16 into
one of its two operands, so its two halves differ by that rounding (2^-9 per
element); both of them enter the sums.  Reversing the electrons exchanges
the halves.  What may change then is the fp32 accumulation (2e-5 of the
largest sum) and single elements whose bf16 rounding turns over: 5e-5."""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ns,G,W,noise", [(64, 16, 64, 4, 0.02), (64, 32, 64, 36, 0.1), (128, 16, 128, 132, 0.05), (128, 32, 128, 20, 0.1)])
def test_reversed_electrons(n, ns, G, W, noise):
    m = inputs.molecule_inputs(n, ns, ns, G, dt=0.005, decay=20.0, seed=7)
    wf, lw, al = inputs.initial_walkers(m.phiTUp, W, seed=3, noise=noise)
    out = []
    for _ in range(2):
        e = capi.pl_engine(m, W, 31, 1000, 1000, precision=capi.AFQMC_MIXED)
        e.set_walkers(wf, lw, al)
        e.reset_measurement()
        e.add_mixed_measurement()
        out.append(e.cholesky_nums()[1] / e.measurement()[0])
        assert e.status() == 0
        e.close()
        m.phiTUp, m.phiTDn, wf = (np.asfortranarray(a[:, ::-1]) for a in (m.phiTUp, m.phiTDn, wf))
    assert np.abs(out[0] - out[1]).max() < 5e-5 * np.abs(out[0]).max()
