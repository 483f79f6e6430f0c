"""The two forms of the ALS-guided Gram-Schmidt against the oracle at the sizes
where their tiles end: the one-cluster form (gs.cu) at ranks 1 to 16 (its
instances for rank 16 and for any rank), bases that take one or two columns
per lane or halves of a warp, fewer and more vectors than CTAs, overlaps in
shared and in global memory; the grid form (gs_grid.cu) with its solve by rows
(rank <= 16) and at ranks around 17, 32, 33 and
64 (slabs of 16 rows, two and four of them); two modes, ragged ranks.  Blocks
of random vectors, npow = 0.

Tolerance.  Both sides solve the same sequence of well-conditioned least-squares
fits, here with 48-bit operands and corrections to 1e-10 of the solution;
1 - cos of the angle between the functions is the square of their distance,
so 1e-10 allows a distance of 1e-5, the bound of the cycle's own tests.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT

CASES = [  # nbas, rank, vectors, sweeps, ragged
    ([5, 4, 6], 1, 4, 2, False),
    ([12, 10], 9, 6, 2, False),
    ([17, 3, 16], 15, 18, 1, True),
    ([33, 32, 6], 16, 5, 1, False),
    ([16, 5, 4], 16, 35, 1, True),
    ([64, 9, 6], 16, 4, 1, False),
    ([3] * 12, 16, 90, 1, False),   # overlaps in global memory
    ([64, 6, 5], 16, 40, 1, True),  # the grid form by rows
    ([18, 9, 7], 17, 6, 2, True),
    ([16, 10, 12], 32, 10, 1, False),
    ([9, 12, 8], 33, 4, 1, True),
    ([12, 13, 10], 64, 4, 1, False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_gram_schmidt_matches_oracle(case, cuda_device):
    nbas, R, B, nals, ragged = CASES[case]
    hl = H.random_hoplist(nbas, 3, seed=20 + case)
    rng = np.random.default_rng(40 + case)
    Q = rng.uniform(-0.5, 0.5, size=(R * B, sum(nbas)))
    qc = rng.uniform(0.5, 1.0, R * B)
    ranks = None
    if ragged:
        ranks = rng.integers(max(1, R // 2), R + 1, B)
        ranks[0] = R
    gb, gc, _ = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, False, 1, 0.0, ranks=ranks)
    if ranks is None:
        ranks = np.full(B, R)
        ob, oc, _ = oracle.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, False, 1, 0.0)
    else:
        live = np.concatenate([np.arange(v * R, v * R + ranks[v]) for v in range(B)])
        ob, oc = oracle.pals_ortho2(Q[live], qc[live], hl.nbas, 0, B, nals, ranks=list(ranks))
    at = 0
    for v in range(B):
        g, o = slice(v * R, v * R + ranks[v]), slice(at, at + ranks[v])
        at += ranks[v]
        gg = oracle.cp_dot(gb[g], gc[g], gb[g], gc[g], nbas)
        oo = oracle.cp_dot(ob[o], oc[o], ob[o], oc[o], nbas)
        go = oracle.cp_dot(gb[g], gc[g], ob[o], oc[o], nbas)
        assert abs(1 - gg) <= 1e-10 and 1 - go / np.sqrt(gg * oo) <= 1e-10, (v, 1 - gg, 1 - go / np.sqrt(gg * oo))
        assert not np.any(gc[v * R + ranks[v]:(v + 1) * R])
