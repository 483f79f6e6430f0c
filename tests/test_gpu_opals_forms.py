"""The two forms of the ALS-fitted Hamiltonian applications, one CTA per
vector (opals.cu) and the grid form (opals_grid.cu), against the oracle at
the sizes where the grid form's tiles end: ranks around 16, 32 and 64 (row
tiles of 16, 32 and two passes of 32), bases around 16, 32, 48 and 64
(column tiles of 16, narrow modes beside wide ones), more and fewer
operators than CTAs, several thousand rows of one right-hand side, ragged
ranks, each sign of the shift.  Three-mode random Hamiltonians; npow = 1 and
no Gram-Schmidt, so that a sweep from a random block is all there is.  Every
rank is below the product of any two bases, so that no normal equations are
singular.

Both forms run the same double-word operations in the same order; against
FP64 a sweep from a random block agrees to the conditioning of its normal
equations (1e-10 as functions is the bound of the power sweep's own tests).
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT

CASES = [  # nbas, rank, vectors, terms, ishift, ragged
    ([17, 5, 9], 16, 3, 9, 1, False),
    ([16, 33, 4], 17, 2, 12, -1, False),
    ([32, 16, 5], 33, 2, 10, 0, False),
    ([48, 31, 15], 32, 2, 30, 1, False),
    ([64, 49, 2], 31, 3, 25, 1, True),
    ([32, 31, 16], 64, 2, 6, 1, True),
    ([6, 5, 7], 15, 40, 400, 1, False),
    ([4, 4, 4], 3, 2, 4, 1, False),   # one CTA per vector
    ([10, 9, 8], 12, 5, 8, -1, True),  # one CTA per vector
    ([6, 5, 6, 6, 6, 7, 6, 6], 20, 2, 12, 1, True),  # one CTA, h_u Fo_j of one mode at a time
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_power_sweep_matches_oracle(case, cuda_device):
    nbas, R, B, T, ishift, ragged = CASES[case]
    hl = H.random_hoplist(nbas, T, seed=60 + case)
    rng = np.random.default_rng(90 + case)
    Q = rng.uniform(-0.5, 0.5, size=(R * B, sum(nbas)))
    qc = rng.uniform(0.5, 1.0, R * B)
    ranks = rng.integers(max(1, R // 3), R + 1, B) if ragged else None
    eig = np.arange(B, dtype=float)
    gb, gc, _ = IT.intertwine(Q, qc, hl.nbas, R, B, hl, eig, 1, 0, False, ishift, 7.5, ranks=ranks)
    for v in range(B):
        r = R if ranks is None else int(ranks[v])
        s = slice(v * R, v * R + r)
        ob, oc, _ = oracle.intertwine(Q[s], qc[s], hl.nbas, r, 1, hl, eig[:1], 1, 0, False, ishift, 7.5)
        gg = oracle.cp_dot(gb[s], gc[s], gb[s], gc[s], nbas)
        oo = oracle.cp_dot(ob, oc, ob, oc, nbas)
        go = oracle.cp_dot(gb[s], gc[s], ob, oc, nbas)
        assert 1 - go / np.sqrt(gg * oo) <= 1e-10, (v, 1 - go / np.sqrt(gg * oo))
        if ranks is not None:
            assert not np.any(gc[v * R + r:(v + 1) * R])
