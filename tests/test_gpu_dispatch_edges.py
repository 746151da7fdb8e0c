"""The far edges of two dispatches, where a shape leaves the panel kernels.

Gram-Schmidt: the panel kernel takes up to 512 rows whose panels and sums fit 227
KB of shared memory (fewer columns for more rows); beyond, one column at a time.
LU: two spin blocks of up to 64 columns share a cluster, up to 120 columns one
thread block's shared memory; beyond, the matrix stays in device memory."""
import numpy as np
import pytest

from afqmclab_b200 import capi
from tests.test_gpu_gram_schmidt import check as check_columns
from tests.test_gpu_gram_schmidt import stabilised, walkers
from tests.test_gpu_lu_block import check as check_blocks
from tests.parity_common import hubbard, molecule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,N", [(15, 16, 48), (16, 16, 40), (14, 16, 200)])
@pytest.mark.parametrize("cond", [1.0, 1e6])
def test_gram_schmidt_of_a_lattice(nx, ny, N, cond):
    h = hubbard(nx=nx, ny=ny, nup=N // 2, ndn=N // 2)
    wf, lw, al = walkers(2 * nx * ny, N, 2, cond, N)
    q, lg = stabilised(capi.cp_engine(h, 2, 1, 1000, 1000), wf, lw, al)
    check_columns(q, lg, wf, lambda lr: lr.sum(), max(np.linalg.cond(wf[:, :, w]) for w in range(2)))


@pytest.mark.parametrize("n", [512, 513])
@pytest.mark.parametrize("cond", [1.0, 1e6])
def test_gram_schmidt_of_a_molecule(n, cond):
    wf, lw, al = walkers(n, 5, 2, cond, n)
    q, lg = stabilised(capi.pl_engine(molecule(n=n, nup=5, ndn=0, G=1), 2, 1, 1000, 1000), wf, lw, al)
    check_columns(q, lg, wf, lambda lr: lr.sum(), max(np.linalg.cond(wf[:, :, w]) for w in range(2)))


@pytest.mark.parametrize("nup,ndn", [(64, 63), (65, 64), (65, 1), (120, 3), (121, 3)])
def test_two_blocks(nup, ndn):
    check_blocks(nup + 5, nup, ndn, 3, 0.3 / (nup + 5) ** 0.5)
