"""The block's H matrix with and without its overlaps (rq.cu): without, the identity of a
mode is left out unless a term has it there, so the matrix must be the same bits;
with terms on every mode, on some, and on none but the identity; against dense vectors
(FP64 sums of at most 1e5 products, so 1e-11 of the largest entry).
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT

NB = [5, 7, 4]


def operators(case):
    rng = np.random.default_rng(case)
    m = {d: (lambda x: x + x.T)(rng.normal(size=(n, n))) for d, n in enumerate(NB)}
    return [[(1.0, m)], [(0.5, {0: m[0], 2: m[2]}), (-1.5, {0: m[2 - 2]})], [(2.0, {1: m[1]}), (1.0, m), (0.3, {2: m[2]})]][case]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(3))
@pytest.mark.parametrize("R,B", [(1, 3), (12, 5), (13, 2)])
def test_matrix_without_overlaps(case, R, B, cuda_device):
    hl = H.build_hoplist(NB, operators(case))
    rng = np.random.default_rng(R)
    Q, qc = rng.uniform(-0.5, 0.5, (R * B, sum(NB))), rng.uniform(0.5, 1.0, R * B)
    a = IT.qhq(Q, qc, NB, R, B, hl)
    b, s = IT.qhq(Q, qc, NB, R, B, hl, overlaps=True)
    np.testing.assert_array_equal(a, b)
    v = np.array([oracle.cp_dense(Q[k * R:(k + 1) * R], qc[k * R:(k + 1) * R], NB).ravel() for k in range(B)])
    h = v @ H.dense_hamiltonian(hl) @ v.T
    assert np.abs(a - h).max() <= 1e-11 * np.abs(h).max()
    assert np.abs(s - v @ v.T).max() <= 1e-11 * np.abs(s).max()
