"""Engines whose background, and with it every one-body operator, is replaced
give what an engine made with the new operators gives: the measurement's half
step and the step's operator both follow."""
import copy

import numpy as np
import pytest

from afqmclab_b200 import capi, inputs

pytestmark = pytest.mark.gpu


def shifted(m):
    m2 = copy.deepcopy(m)
    m2.set_background(0.3 * np.cos(np.arange(m.G)))
    return m2


def outputs(e, m):
    wf, lw, al = inputs.initial_walkers(m.phiTUp, e.W, seed=82, noise=0.02)
    e.set_walkers(wf, lw, al)
    e.set_rng(81)
    e.reset_measurement()
    e.add_mixed_measurement()
    s = e.measurement()
    e.step(1)
    out = [s[:2], *e.cholesky_nums(), e.get_walkers()[0], e.log_overlaps()]
    assert e.status() == 0
    e.close()
    return out


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("prec", [capi.AFQMC_FP64, capi.AFQMC_MIXED])
def test_update_equals_a_new_engine(prec, graphs):
    m = inputs.molecule_inputs(64, 16, 16, 128, dt=0.005, decay=30.0, seed=7)
    m.ET = -5.0
    m2 = shifted(m)
    e = capi.pl_engine(m, 12, 81, 1000, 1000, precision=prec)
    e.set_graphs(graphs)
    wf, lw, al = inputs.initial_walkers(m.phiTUp, 12, seed=82, noise=0.02)
    e.set_walkers(wf, lw, al)
    for _ in range(3):
        e.step(1)
        e.add_mixed_measurement()
    e.update_background(m2)
    for a, b in zip(outputs(e, m2), outputs(capi.pl_engine(m2, 12, 81, 1000, 1000, precision=prec), m2)):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * np.abs(b).max())


def test_real_and_complex_operators_take_turns():
    """The FP64 form multiplies by real copies of real operators; graphs captured
    with them are dropped when the operators change to complex ones and back."""
    m = inputs.molecule_inputs(40, 9, 7, 24, dt=0.005, decay=6.0, seed=7)
    m.ET = -5.0
    rng = np.random.default_rng(3)
    x = rng.standard_normal((m.n, m.n))
    mc = shifted(m)
    for name in ("expMinusDtK", "expHalfDtK", "expMinusHalfDtK"):
        setattr(mc, name, np.asfortranarray(getattr(mc, name) + 1e-3j * (x - x.T)))
    e = capi.pl_engine(m, 12, 81, 1000, 1000)
    e.set_graphs(True)
    for m2 in (m, mc, m, mc):
        e.update_background(m2)
        wf, lw, al = inputs.initial_walkers(m.phiTUp, 12, seed=82, noise=0.02)
        out = []
        for f in (e, capi.pl_engine(m2, 12, 81, 1000, 1000)):
            f.set_walkers(wf, lw, al)
            f.set_rng(81)
            for _ in range(3):   # direct, captured, replayed
                f.reset_measurement()
                f.add_mixed_measurement()
                f.step(1)
            out.append([f.measurement()[:2], f.get_walkers()[0], f.log_overlaps()])
        f.close()
        for a, b in zip(*out):
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * np.abs(b).max())
    assert e.status() == 0
    e.close()
