"""Rayleigh quotients (rq.cu) by one CTA and by clusters of up to eight that share a
vector's columns: ranks below, at and above the cluster's size, ranks that do
not divide by it, few vectors (eight CTAs each) and more vectors than SMs (one each),
against the oracle.  Both are FP64 and differ in the order of their sums: of
R^2 T products of up to D + 2 factors, each within (D + n) 2^-53, so 1e-11
relative allows for cancellation by 1e3.  However the vectors are dealt to
clusters, every sum keeps its order: the same vectors in a larger block give the
same bits.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT

CASES = [  # nbas, rank, vectors, nconv
    ([5, 7, 4], 1, 3, 0),
    ([6, 5], 3, 2, 1),
    ([4, 9, 6, 3], 8, 1, 0),
    ([10, 8, 5], 13, 25, 2),
    ([12, 5, 7], 33, 80, 40),
    ([4, 3, 5], 6, 160, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_rayleigh_quotients(case, cuda_device):
    nbas, R, B, nconv = CASES[case]
    hl = H.random_hoplist(nbas, 6, seed=case)
    rng = np.random.default_rng(case)
    Q = rng.uniform(-0.5, 0.5, size=(R * B, sum(nbas)))
    qc = rng.uniform(0.1, 1.0, R * B)
    got = IT.qhq_diag(Q, qc, hl.nbas, R, B, hl, nconv=nconv)
    want = oracle.qhq_diag(Q, qc, hl.nbas, R, B, hl, nconv)
    np.testing.assert_allclose(got[nconv:], want[nconv:], rtol=1e-11)
    last = IT.qhq_diag(Q, qc, hl.nbas, R, B, hl, nconv=B - 1)  # one vector: the largest cluster
    assert last[B - 1] == got[B - 1]
