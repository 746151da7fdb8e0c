"""The FP64 form's choice of products by the operators' values, against the
oracle to 1e-10 per step.

Real one-body operators and trials take real products; a trial whose first
columns live on the spin-up rows and the others on the spin-down rows, and
one-body operators without entries between the spins, take each spin by
itself; symmetric Cholesky vectors give the two-body matrix as panels of
its lower triangle.  Each form is checked next to the general one: complex
values, mixed spins, columns in another order, vectors that are not symmetric.
"""
import numpy as np
import pytest

from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, compare_state, hubbard, molecule, pair_cp, pair_pl

pytestmark = pytest.mark.gpu


def check(g, o, seed, sums):
    for _ in range(2):
        wf, lw, al = o.get_walkers()
        g.set_walkers(wf, lw, al)
        g.set_rng(seed, o.rng_counter())
        g.step(1)
        o.step(1)
        compare_state(g, o, STEP_TOL)
        assert rel_err(g.get_walkers()[0], o.get_walkers()[0]) < STEP_TOL
    wf, lw, al = o.get_walkers()
    g.set_walkers(wf, lw, al)
    for e in (g, o):
        e.reset_measurement()
        e.add_mixed_measurement()
    mg, mo = g.measurement(), o.measurement()
    assert rel_err(mg[:2], mo[:2]) < STEP_TOL
    for k in range(2, sums):
        assert abs(mg[k] - mo[k]) <= STEP_TOL * max(1.0, abs(mo[1]))
    assert rel_err(g.green(0), o.green(0)) < STEP_TOL
    assert logov_close(g.log_overlaps(), o.log_overlaps(), STEP_TOL) < STEP_TOL


def hubbard_form(decomp, form):
    m = hubbard(decomp, False, nx=3, ny=4, nup=5, ndn=4)
    rng = np.random.default_rng(11)
    if form == "complex trial":
        m.phiT = np.asfortranarray(m.phiT * np.exp(1j * rng.uniform(-0.3, 0.3, m.N))[None, :])
    elif form == "columns shuffled":
        m.phiT = np.asfortranarray(m.phiT[:, rng.permutation(m.N)])
    elif form == "spin-down first":
        m.phiT = np.asfortranarray(np.roll(m.phiT, m.ndn, axis=1))
    elif form == "spins mixed":
        x = rng.standard_normal((m.n, m.n)) + 1j * rng.standard_normal((m.n, m.n))
        m.K = np.asfortranarray(m.K + 0.1 * (x + x.conj().T))
        lam, v = np.linalg.eigh(m.K)
        for name, a in (("expMinusDtK", m.dt), ("expHalfDtK", -0.5 * m.dt), ("expMinusHalfDtK", 0.5 * m.dt)):
            setattr(m, name, np.asfortranarray((v * np.exp(-a * lam)) @ v.conj().T))
    elif form == "one spin":
        m = hubbard(decomp, False, nx=3, ny=4, nup=5, ndn=0)
    return m


@pytest.mark.parametrize("decomp", ["densityCharge", "densitySpin", "hopCharge", "hopSpin"])
@pytest.mark.parametrize("form", ["plain", "complex trial", "columns shuffled", "spin-down first", "spins mixed", "one spin"])
def test_hubbard_forms(decomp, form):
    g, o = pair_cp(hubbard_form(decomp, form), 5, 77, 1000, 1000)
    check(g, o, 77, 5)


@pytest.mark.parametrize("n,nup,ndn", [(9, 3, 3), (16, 5, 2), (40, 17, 9)])
@pytest.mark.parametrize("form", ["complex trial", "complex operators", "not symmetric"])
def test_molecule_forms(form, n, nup, ndn):
    m = molecule(n=n, nup=nup, ndn=ndn, G=11)
    rng = np.random.default_rng(12)
    if form == "complex trial":
        m.phiTUp = np.asfortranarray(m.phiTUp * np.exp(0.2j))
        m.phiTDn = np.asfortranarray(m.phiTDn * np.exp(-0.1j))
    elif form == "complex operators":
        x = rng.standard_normal((n, n))
        for name in ("expMinusDtK", "expHalfDtK", "expMinusHalfDtK"):
            setattr(m, name, np.asfortranarray(getattr(m, name) + 1e-3j * (x - x.T)))
    else:
        m.chol = np.asfortranarray(m.chol.copy())
        m.chol[n - 1, 0, 3] += 0.01
    g, o = pair_pl(m, 4, 78, 1000, 1000)
    check(g, o, 78, 3)


@pytest.mark.parametrize("decomp", ["densitySpin", "densityCharge", "hopSpin"])
@pytest.mark.parametrize("nx,ny,fields", [(4, 8, False), (3, 11, False), (8, 8, True), (5, 13, False), (8, 16, False), (3, 43, False)])
def test_sample_in_the_one_body_product(decomp, nx, ny, fields):
    """A diagonal sample scales the one-body product's rows, in place where one
    tile holds them (32, 64 and 128 sites are the tiles' ends); transverse
    fields, hopping decompositions and larger lattices apply it on its own."""
    m = hubbard(decomp, fields, nx=nx, ny=ny, nup=5, ndn=4)
    g, o = pair_cp(m, 3, 79, 1000, 1000)
    check(g, o, 79, 5)


def test_dead_walkers_and_many_walkers_draw_from_their_own_place():
    """The place in the random stream counts the survivors before a walker, in
    the sampling kernel up to 4096 walkers and by the scan above."""
    m = hubbard("densitySpin", False, nx=2, ny=2, nup=1, ndn=1)
    for W in (7, 4096, 4097):
        g, o = pair_cp(m, W, 80, 1000, 1000)
        wf, lw, al = o.get_walkers()
        al[::3] = 0
        o.set_walkers(wf, lw, al)
        g.set_walkers(wf, lw, al)
        for _ in range(2):
            g.step(1)
            o.step(1)
            compare_state(g, o, STEP_TOL)
