"""The mixed form's exchange as half products of symmetric quadratic forms:
block counts of K = Ns n / 256 from 2 to 16, one and two spin blocks, walker
numbers that do not fill a tile.  Against the FP64 form on the same walkers,
to the bf16 operands' accuracy (energies 2e-3, per-vector sums 2e-2)."""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nup,ndn,G,W", [(64, 16, 16, 64, 4), (64, 48, 32, 64, 36), (128, 16, 16, 192, 132), (128, 48, 48, 64, 20)])
def test_energy_and_vector_sums(n, nup, ndn, G, W):
    m = inputs.molecule_inputs(n, nup, ndn, G, dt=0.005, decay=20.0, seed=7)
    wf, lw, al = inputs.initial_walkers(m.phiTUp, W, seed=3, noise=0.02)
    out = []
    for prec in (capi.AFQMC_FP64, capi.AFQMC_MIXED):
        e = capi.pl_engine(m, W, 31, 1000, 1000, precision=prec)
        e.set_walkers(wf, lw, al)
        e.reset_measurement()
        e.add_mixed_measurement()
        s = e.measurement()
        out.append((s[1] / s[0], e.cholesky_nums()))
        assert e.status() == 0
        e.close()
    (ef, (bf, xf)), (ex, (bx, xx)) = out
    assert abs(ef - ex) < 2e-3 * abs(ef)
    assert np.abs(bf - bx).max() < 2e-2 * np.abs(bf).max()
    assert np.abs(xf - xx).max() < 2e-2 * np.abs(xf).max()
