"""modifyGM (Gram-Schmidt) at the edges of its rows per warp, panels and
storage, against numpy's QR with a positive diagonal.

32 rows per warp, panels of 8 columns, finished panels in shared memory or read
back from memory (above 40 KB per walker), one thread block up to 448 rows.  The
walkers' columns have condition numbers up to 1e6: modified Gram-Schmidt
keeps Q^H Q - 1 within a small multiple of cond * eps, and Q R equals the walker
to rounding.
"""
import numpy as np
import pytest

from afqmclab_b200 import capi, inputs
from tests.parity_common import hubbard, molecule

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def stabilised(e, wf, lw, al):
    e.set_walkers(wf, lw, al)
    e.modify_gm()
    q, lg, _ = e.get_walkers()
    assert e.status() == 0
    e.close()
    return q, lg


def check(q, lg, wf, factor, cond, eps=EPS):
    n, N, W = wf.shape
    for w in range(W):
        Q, R = np.linalg.qr(wf[:, :, w])
        d = np.diag(R)
        tol = 20 * N * cond * eps
        assert np.abs(q[:, :, w].conj().T @ q[:, :, w] - np.eye(N)).max() < tol
        # the span and the gauge: Q^H of numpy's with the phases of its diagonal
        assert np.abs(q[:, :, w] - Q * (d / np.abs(d))[None, :]).max() < tol
        assert abs(lg[w].real - factor(np.log(np.abs(d)))) < tol * N


def walkers(n, N, W, cond, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, N, W)) + 1j * rng.standard_normal((n, N, W))
    if cond > 1.0:   # every column close to the first one
        a = a / cond + a[:, :1]
    return np.asfortranarray(a), np.zeros(W, np.complex128), np.ones(W, np.int32)


@pytest.mark.parametrize("n,N", [(1, 1), (7, 3), (8, 8), (31, 9), (32, 16), (33, 17), (64, 7), (65, 64), (96, 40),
                                 (128, 33), (160, 63), (257, 18), (288, 121), (448, 10), (449, 5)])
@pytest.mark.parametrize("cond", [1.0, 1e6])
def test_molecule(n, N, cond):
    m = molecule(n=n, nup=N, ndn=0, G=1)
    wf, lw, al = walkers(n, N, 3, cond, n + N)
    c = max(np.linalg.cond(wf[:, :, w]) for w in range(3))
    q, lg = stabilised(capi.pl_engine(m, 3, 1, 1000, 1000), wf, lw, al)
    check(q, lg, wf, lambda lr: lr.sum(), c)


def test_two_spins_and_lattice():
    m = molecule(n=40, nup=11, ndn=6, G=1)
    wf, lw, al = walkers(40, 11, 2, 1.0, 5)
    q, lg = stabilised(capi.pl_engine(m, 2, 1, 1000, 1000), wf, lw, al)
    check(q, lg, wf, lambda lr: lr.sum() + lr[:6].sum(), 10.0)
    h = hubbard(nx=4, ny=5, nup=9, ndn=8)
    wf, lw, al = walkers(40, 17, 2, 1.0, 6)
    q, lg = stabilised(capi.cp_engine(h, 2, 1, 1000, 1000), wf, lw, al)
    check(q, lg, wf, lambda lr: lr.sum(), 10.0)


@pytest.mark.parametrize("n,N", [(64, 16), (64, 48), (128, 32), (128, 64)])
def test_mixed(n, N):
    m = molecule(n=n, nup=N, ndn=N, G=64)
    wf, lw, al = inputs.initial_walkers(m.phiTUp, 3, seed=9, noise=0.02)
    wf = np.asfortranarray(wf.astype(np.complex64).astype(np.complex128))
    e = capi.pl_engine(m, 3, 1, 1000, 1000, precision=capi.AFQMC_MIXED)
    q, lg = stabilised(e, wf, lw, al)
    check(q, lg, wf, lambda lr: 2 * lr.sum(), 1.0, eps=2.0 ** -24 / N)   # columns rounded to fp32 once
