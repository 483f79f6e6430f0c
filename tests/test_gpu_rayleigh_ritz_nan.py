"""The generalised eigensolver of the Rayleigh-Ritz step (gep.cu) on a Hamiltonian that
is not finite.
"""
import numpy as np
import pytest

from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT


@pytest.mark.gpu
@pytest.mark.parametrize("nbas", [[2, 2, 2], [3, 4, 3]])
def test_nan_in_the_hamiltonian_reaches_every_eigenvalue(nbas, cuda_device):
    """A Hamiltonian with a NaN gives NaN eigenvalues, not what an earlier call left in the
    workspace (three modes and nals = 0: eigenvalues only)."""
    B = int(np.prod(nbas))
    base, coef = np.zeros((B, sum(nbas))), np.ones(B)
    for v, ix in enumerate(np.ndindex(*nbas)):
        base[v, [sum(nbas[:d]) + i for d, i in enumerate(ix)]] = 1.0
    hl = H.random_hoplist(nbas, 5, 3)
    _, _, ge = IT.diagonalize(base, coef, hl.nbas, 1, B, hl, 0)
    assert np.all(np.isfinite(ge))
    hl.coef = np.array(hl.coef, dtype=np.float64)
    hl.coef[0] = np.nan
    _, _, ge = IT.diagonalize(base, coef, hl.nbas, 1, B, hl, 0)
    assert np.all(np.isnan(ge))
