"""The pivot search of the LU compares all 64 bits of |re| + |im|.

Rows i < j of the overlap matrix hold 1 and 1 + 2^-30 in column i, and the
largest finite number X and 0 in column j; the rest is the identity.  zgetf2
takes row j and leaves X as the other pivot.  An elimination that took row i
would multiply X by 1 + 2^-30, which overflows.  The sizes put the rows in
one warp, in two warps and in two thread blocks, in panels and in the
element-wise kernel (25 to 32 columns, more than 888 matrices).

Hadamard matrices tie in every step and take the first position; their
log-determinants and inverses are compared with the oracle's."""
import numpy as np
import pytest
from scipy.linalg import hadamard

from afqmclab_b200 import capi
from tests.helpers import logov_close, rel_err
from tests.parity_common import STEP_TOL, molecule, pair_pl

pytestmark = pytest.mark.gpu
X = np.finfo(float).max


@pytest.mark.parametrize("N,i,j,W", [(2, 0, 1, 2), (16, 7, 8, 2), (20, 3, 17, 2), (27, 2, 26, 889), (40, 5, 20, 2), (40, 5, 38, 2),
                                     (64, 31, 63, 2), (70, 10, 66, 2), (128, 31, 96, 2), (128, 65, 127, 2)])
@pytest.mark.parametrize("phase", [1.0, -1j])
def test_near_ties(N, i, j, W, phase):
    m = molecule(n=N + 1, nup=N, ndn=0, G=2)
    m.phiTUp = np.asfortranarray(np.eye(N + 1, N).astype(np.complex128))
    S = np.eye(N + 1, N).astype(np.complex128)
    S[i, i], S[j, i], S[i, j], S[j, j] = phase, phase * (1.0 + 2.0 ** -30), X, 0.0
    e = capi.pl_engine(m, W, 3, 1000, 1000)
    e.set_walkers(np.asfortranarray(np.repeat(S[:, :, None], W, axis=2)), np.zeros(W, np.complex128), np.ones(W, np.int32))
    lo = e.log_overlaps() - np.conj(m.logwT)
    det = -phase   # times X (1 + 2^-30)
    assert np.abs(lo.real - (np.log1p(2.0 ** -30) + np.log(X))).max() < 1e-12
    assert np.abs(np.exp(1j * lo.imag) - det).max() < 1e-12
    assert e.status() == 0
    e.close()


@pytest.mark.parametrize("N,W", [(2, 2), (16, 2), (32, 2), (32, 889), (64, 2), (128, 2)])
def test_equal_entries(N, W):
    m = molecule(n=N + 2, nup=N, ndn=0, G=2)
    m.phiTUp = np.asfortranarray(np.eye(N + 2, N).astype(np.complex128))
    wf = np.zeros((N + 2, N, W), np.complex128, order="F")
    wf[:N] = hadamard(N)[:, :, None] * np.exp(1j * np.linspace(0.0, 1.0, W))
    wf[N:] = 0.5
    g, o = pair_pl(m, W, 4, 1000, 1000)
    lw, al = np.zeros(W, np.complex128), np.ones(W, np.int32)
    for e in (g, o):
        e.set_walkers(wf, lw, al)
    assert logov_close(g.log_overlaps(), o.log_overlaps(), STEP_TOL) < STEP_TOL
    for w in (0, W - 1):
        assert rel_err(g.green(w), o.green(w)) < STEP_TOL
