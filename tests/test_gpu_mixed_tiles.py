"""Overlap and theta tiles of the mixed form: walker numbers around the tile
choices (one walker a tile, several, a last tile in part), block widths that
are no multiple of 16, blocks whose inverses do not start on 16 bytes, one and
two blocks per launch.  Against the FP64 form from the same walkers: fp32
walkers and tf32 pairs leave 2^-21 of each overlap element, so log-overlaps
agree to 2 Ns 2^-21 < 1e-4; the force sums carry bf16 operands (2e-2)."""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nup,ndn,W", [
    (64, 16, 16, 1), (64, 32, 17, 149), (64, 32, 20, 700), (64, 16, 16, 2500),
    (128, 64, 33, 297), (128, 48, 40, 310), (128, 64, 64, 150)])
def test_overlap_and_theta_match_fp64(n, nup, ndn, W):
    m = inputs.molecule_inputs(n, nup, ndn, 64, dt=0.005, decay=20.0, seed=7)
    wf, lw, al = inputs.initial_walkers(m.phiTUp, W, seed=3, noise=0.02)
    out = []
    for prec in (capi.AFQMC_FP64, capi.AFQMC_MIXED):
        e = capi.pl_engine(m, W, 31, 1000, 1000, precision=prec)
        e.set_walkers(wf, lw, al)
        lo = e.log_overlaps()
        e.reset_measurement()
        e.add_mixed_measurement()
        out.append((lo, e.cholesky_nums()))
        assert e.status() == 0
        e.close()
    (lf, (bf, xf)), (lx, (bx, xx)) = out
    assert np.abs(lf - lx).max() < 1e-4
    assert np.abs(bf - bx).max() < 2e-2 * np.abs(bf).max()
    assert np.abs(xf - xx).max() < 2e-2 * np.abs(xf).max()
