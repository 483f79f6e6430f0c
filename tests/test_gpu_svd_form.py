"""The dense matrix of the two-mode SVD at the edges of its staging: 64 mode-1 indices of a
block of 256 entries are staged, 65 are not; transposed matrices whose blocks span
one, two or many columns; terms that fill their stages of 32 or not; the last block
partial.  Checks and tolerances as in test_gpu_svd.py.
"""
import numpy as np
import pytest

from mlcp_gb300 import intertwine as IT
from test_gpu_svd import check, make_batch

CASES = [([64, 5], 33), ([65, 5], 31), ([64, 64], 32), ([66, 65], 65), ([3, 300], 40), ([5, 256], 64), ([2, 90], 1),
         ([40, 40], 96)]


@pytest.mark.gpu
@pytest.mark.parametrize("nbas,rG", CASES)
def test_staged_matrix(nbas, rG, cuda_device):
    rng = np.random.default_rng(rG)
    base, coef = make_batch(rng, 2, rG, nbas)
    gb, gc, gr = IT.reduc_svd(base.reshape(-1, sum(nbas)), coef.ravel(), nbas, rG, 4)
    check(gb, gc, gr, base, coef, nbas, 4)
