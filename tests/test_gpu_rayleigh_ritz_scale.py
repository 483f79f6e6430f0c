"""The generalised eigensolver of the Rayleigh-Ritz step (gep.cu) on Hamiltonians in
units far from one.
"""
import numpy as np
import pytest

from mlcp_gb300 import intertwine as IT
from test_gpu_rayleigh_ritz import operators, product_block


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2", [(2, 3), (5, 5), (12, 12)])
@pytest.mark.parametrize("power", [-140, -100, 80, 120])
def test_power_of_two_only_scales(n1, n2, power, cuda_device):
    """Every operation of the solver is linear in H or free of its scale, so a power of two
    in front of H is one in front of the eigenvalues, and no other bit changes; also where
    H or its squares leave the range of FP32."""
    B, rk = n1 * n2, min(n1, n2)
    base, coef = product_block(n1, n2, rk)
    out = []
    for p in (0, power):
        hl = operators("field", n1, n2)
        hl.coef = np.ldexp(np.asarray(hl.coef, dtype=np.float64), p)
        out.append(IT.diagonalize(base, coef, hl.nbas, rk, B, hl, 0))
    np.testing.assert_array_equal(out[1][2], np.ldexp(out[0][2], power))
    np.testing.assert_array_equal(out[1][0], out[0][0])
    np.testing.assert_array_equal(out[1][1], out[0][1])
