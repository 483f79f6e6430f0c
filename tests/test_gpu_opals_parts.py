"""ALS-fitted Hamiltonian applications of a block whose scratch does not fit the bound for
one launch: the block goes through in parts.  Vectors do not depend on one another,
so the result is the same bits as for the parts' vectors in calls of their own.  (420
vectors of rank 30, three modes of 48 functions, 1000 terms: 42 MB a vector against 16 GB;
ragged ranks, so that the parts' offsets matter in every argument.)
"""
import numpy as np
import pytest

from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT


@pytest.mark.gpu
def test_block_in_parts(cuda_device):
    nb, R, B = [48, 48, 48], 30, 420
    hl = H.random_hoplist(nb, 1000, 3)
    rng = np.random.default_rng(4)
    Q, c = rng.uniform(-0.5, 0.5, size=(B * R, sum(nb))), rng.uniform(0.5, 1.0, B * R)
    ranks = rng.integers(8, R + 1, B)
    run = lambda v0, v1: IT.intertwine(Q[v0 * R:v1 * R], c[v0 * R:v1 * R], hl.nbas, R, v1 - v0, hl,  # noqa: E731
                                       np.zeros(v1 - v0), 1, 0, False, 1, 5.0, ranks=ranks[v0:v1])
    whole = run(0, B)
    for v0, v1 in ((0, 210), (210, B)):
        part = run(v0, v1)
        np.testing.assert_array_equal(whole[0][v0 * R:v1 * R], part[0])
        np.testing.assert_array_equal(whole[1][v0 * R:v1 * R], part[1])
