"""The largest lattices whose sampling kernel fits its 48 KB of shared memory: 646
sites in the FP64 form, 818 (an even number) in the mixed form.  FP64 against the
oracle to 1e-10 per step, the mixed form's log-overlaps to its single-precision
propagation (1e-4)."""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs
from oracle import oracle as O
from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, compare_state, hubbard, pair_cp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("decomp", ["densitySpin", "hopCharge"])
@pytest.mark.parametrize("nx,ny", [(4, 161), (3, 215), (2, 323)])
def test_fp64(decomp, nx, ny):
    m = hubbard(decomp, False, nx=nx, ny=ny, nup=1, ndn=1)
    g, o = pair_cp(m, 2, 92, 1000, 1000)
    g.step(1)
    o.step(1)
    compare_state(g, o, STEP_TOL)
    assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL


@pytest.mark.parametrize("nx,ny", [(2, 408), (2, 409)])
def test_mixed(nx, ny):
    m = hubbard("densitySpin", False, nx=nx, ny=ny, nup=2, ndn=2)
    wf, lw, al = inputs.initial_walkers(m.phiT, 4, seed=6, noise=0.002)
    g = capi.cp_engine(m, 4, 93, 1000, 1000, precision=capi.AFQMC_MIXED)
    o = O.cp_engine(m, 4, 93, 1000, 1000)
    for e in (g, o):
        e.set_walkers(wf, lw, al)
        e.step(1)
    assert g.status() == 0
    assert np.array_equal(g.get_walkers()[2], o.get_walkers()[2]) and g.get_walkers()[2].all()
    assert logov_close(g.log_overlaps(), o.log_overlaps(), 1e-4) < 1e-4
