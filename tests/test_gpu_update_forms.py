"""The vector updates (upd_grid.cu: right-hand sides over ranges of the block's terms,
a solve per vector, overlaps as one matrix product; upd.cu: a cluster per vector, for
small blocks) against the oracle at the sizes where their tiles end: block terms around 64 (overlap tiles) and 32
(stages of a right-hand side), ranks around 16 and 32 (rows of a CTA: 16, 32,
two times 32), bases around 16, 32, 48 and 64 (columns of a thread), more
ranges than one, two modes, ragged ranks.  npow = 0, one or two sweeps of the
orthogonalisation, then the Rayleigh-Ritz problem and the update.

Tolerance: that of the cycle's tests with update, 1 - cos <= 1e-6 and 1e-6 of the
eigenvalues: the Ritz vectors of a random block lie 1e-2 and more apart, so
the stage amplifies the fits' 1e-10 by no more than 1e3 or so.  Ragged blocks with
update read another triangle than the oracle's ragged solver; they are checked
against the same block at equal rank, whose extra terms have no weight.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT

CASES = [  # nbas, rank, vectors, sweeps
    ([17, 6, 5], 16, 4, 2),
    ([16, 33, 4], 13, 5, 1),
    ([49, 7, 18], 17, 3, 1),
    ([64, 9, 48], 32, 2, 1),
    ([12, 13, 11], 33, 4, 1),
    ([32, 12, 7], 3, 43, 1),
    ([9, 8], 5, 13, 2),              # a cluster of four CTAs per vector
    ([6, 7, 5, 4], 6, 60, 1),        # clusters of two
    ([6, 5, 7], 3, 100, 2),          # one CTA per vector
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(CASES)))
def test_update_matches_oracle(case, cuda_device):
    nbas, R, B, nals = CASES[case]
    hl = H.random_hoplist(nbas, 5, seed=30 + case)
    rng = np.random.default_rng(50 + case)
    Q = rng.uniform(-0.5, 0.5, size=(R * B, sum(nbas)))
    qc = np.ones(R * B)
    gb, gc, ge = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, True, 1, 0.0)
    ob, oc, oe = oracle.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, True, 1, 0.0)
    np.testing.assert_allclose(ge, oe, rtol=1e-6, atol=1e-12)
    for v in range(B):
        s = slice(v * R, (v + 1) * R)
        gg = oracle.cp_dot(gb[s], gc[s], gb[s], gc[s], nbas)
        oo = oracle.cp_dot(ob[s], oc[s], ob[s], oc[s], nbas)
        go = oracle.cp_dot(gb[s], gc[s], ob[s], oc[s], nbas)
        assert 1 - abs(go) / np.sqrt(gg * oo) <= 1e-6, (v, 1 - abs(go) / np.sqrt(gg * oo))


@pytest.mark.gpu
@pytest.mark.parametrize("R,extra", [(9, 7), (14, 5), (20, 20)])
def test_ragged_update_ignores_padding(R, extra, cuda_device):
    nbas, B = [9, 12, 8], 5
    hl = H.random_hoplist(nbas, 5, seed=3)
    rng = np.random.default_rng(R)
    Q = rng.uniform(-0.5, 0.5, size=(B, R, sum(nbas)))
    wide = rng.uniform(-0.5, 0.5, size=(B, R + extra, sum(nbas)))
    wide[:, :R] = Q
    a = IT.intertwine(Q.reshape(B * R, -1), np.ones(B * R), hl.nbas, R, B, hl, np.zeros(B), 0, 1, True, 1, 0.0)
    wc = np.zeros((B, R + extra))
    wc[:, :R] = 1.0
    b = IT.intertwine(wide.reshape(B * (R + extra), -1), wc.reshape(-1), hl.nbas, R + extra, B, hl, np.zeros(B), 0, 1, True,
                      1, 0.0, ranks=[R] * B)
    np.testing.assert_allclose(b[2], a[2], rtol=1e-9)
    for v in range(B):
        s, t = slice(v * R, (v + 1) * R), slice(v * (R + extra), v * (R + extra) + R)
        aa = oracle.cp_dot(a[0][s], a[1][s], a[0][s], a[1][s], nbas)
        bb = oracle.cp_dot(b[0][t], b[1][t], b[0][t], b[1][t], nbas)
        ab = oracle.cp_dot(a[0][s], a[1][s], b[0][t], b[1][t], nbas)
        assert 1 - abs(ab) / np.sqrt(aa * bb) <= 1e-6
        assert not np.any(b[1][v * (R + extra) + R:(v + 1) * (R + extra)])
