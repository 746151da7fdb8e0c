"""Walkers handed over by the mixed forms come from their single-precision
planes: the record of any list of walkers (one, several out of order, one
twice) holds the bits that get_walkers and a single walker's copy give."""
import numpy as np
import pytest
import torch

from afqmclab_b200 import capi, inputs
from tests.parity_common import hubbard

pytestmark = pytest.mark.gpu


def engine(kind):
    if kind == "phaseless":
        m = inputs.molecule_inputs(64, 16, 16, 64, dt=0.005, decay=20.0, seed=7)
        wf, lw, al = inputs.initial_walkers(m.phiTUp, 9, seed=3, noise=0.02)
        e = capi.pl_engine(m, 9, 31, 1000, 1000, precision=capi.AFQMC_MIXED)
    else:
        m = hubbard("densitySpin", False, nx=4, ny=4, nup=7, ndn=7)
        wf, lw, al = inputs.initial_walkers(m.phiT, 9, seed=3, noise=0.02)
        e = capi.cp_engine(m, 9, 31, 1000, 1000, precision=capi.AFQMC_MIXED)
    e.set_walkers(wf, lw, al)
    e.step(2)
    return e


@pytest.mark.parametrize("kind", ["phaseless", "constrained"])
@pytest.mark.parametrize("idx", [[4], [8, 0, 3], [5, 5, 1, 7, 6, 5], list(range(9))])
def test_records(kind, idx):
    e = engine(kind)
    wf, lw, _ = e.get_walkers()
    size = e.walker_bytes() // 16
    buf = torch.zeros(len(idx), size, dtype=torch.complex128, device="cuda")
    one = torch.zeros(size, dtype=torch.complex128, device="cuda")
    e.pack_walkers(idx, buf.data_ptr())
    rec = buf.cpu().numpy()
    for k, w in enumerate(idx):
        e.copy_walker_out(w, one.data_ptr())
        assert (rec[k] == one.cpu().numpy()).all()
        assert (rec[k, :-1] == wf[:, :, w].reshape(-1, order="F")).all()
        assert rec[k, -1] == lw[w]
    e.close()
