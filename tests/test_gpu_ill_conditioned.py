"""The Gram-Schmidt and the power sweep on vectors whose terms are nearly the same (as
power iteration leaves them): normal equations of condition 1e6 to 1e8, where the
FP32 inverse is no use and every form falls back to the double-word LDL^T; the forms of the
Gram-Schmidt against one another; and one-mode blocks.

Tolerance.  A solve of condition 1e8 in 48-bit arithmetic (3.6e-15) leaves the weights along
the weak directions right to 4e-7, and these carry little of the function; the
FP64 oracle leaves less.  Half a dozen such steps, each starting from the factors of the
one before, stay far within the distance of 1e-5 (1 - cos <= 1e-10) that the forms'
tests on easy blocks allow.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT


def close_terms(nbas, R, B, eps, seed):
    rng = np.random.default_rng(seed)
    nD = sum(nbas)
    Q = rng.uniform(-0.5, 0.5, size=(B, 1, nD)) + eps * rng.uniform(-0.5, 0.5, size=(B, R, nD))
    return Q.reshape(B * R, nD), rng.uniform(0.5, 1.0, B * R)


def first_condition(Q, nbas, R):
    """Condition of vector 1's normal equations of mode 0 with the reference's penalty."""
    off, G = np.cumsum([0] + list(nbas)), np.ones((R, R))
    for d in range(1, len(nbas)):
        q = Q[R:2 * R, off[d]:off[d + 1]]
        G = G * (q @ q.T)
    return np.linalg.cond(G + 1e-10 * np.eye(R))


def assert_same_functions(gb, gc, ob, oc, nbas, R, B, Ro=None):
    Ro = Ro or R
    for v in range(B):
        g, o = slice(v * R, (v + 1) * R), slice(v * Ro, (v + 1) * Ro)
        gg = oracle.cp_dot(gb[g], gc[g], gb[g], gc[g], nbas)
        oo = oracle.cp_dot(ob[o], oc[o], ob[o], oc[o], nbas)
        go = oracle.cp_dot(gb[g], gc[g], ob[o], oc[o], nbas)
        assert 1 - go / np.sqrt(gg * oo) <= 1e-10, (v, 1 - go / np.sqrt(gg * oo))


GS = [  # nbas, rank, vectors, distance of the terms
    ([10] * 6, 16, 5, 1e-3),       # one cluster, the instance for rank 16
    ([12, 11, 10, 9], 9, 5, 1e-3),  # one cluster, any rank
    ([64, 6, 5], 16, 40, 0.05),    # the grid form by rows
    ([10] * 6, 24, 4, 1e-3),       # the grid form
    ([10] * 6, 40, 3, 1e-2),       # the grid form, the inverse by eight warps
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(GS)))
def test_gram_schmidt_of_close_terms(case, cuda_device):
    nbas, R, B, eps = GS[case]
    Q, qc = close_terms(nbas, R, B, eps, 70 + case)
    assert 1e6 <= first_condition(Q, nbas, R) <= 1e8
    hl = H.random_hoplist(nbas, 3, seed=case)
    gb, gc, _ = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, 1, False, 1, 0.0)
    ob, oc, _ = oracle.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, 1, False, 1, 0.0)
    assert_same_functions(gb, gc, ob, oc, nbas, R, B)


POW = [  # nbas, rank, vectors, terms of H
    ([10] * 6, 16, 3, 11),   # one CTA per vector
    ([24, 22, 23, 20], 20, 3, 60),  # the grid form
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(POW)))
def test_power_sweep_of_close_terms(case, cuda_device):
    nbas, R, B, T = POW[case]
    Q, qc = close_terms(nbas, R, B, 1e-3, 80 + case)
    assert 1e6 <= first_condition(Q, nbas, R) <= 1e8
    hl = H.random_hoplist(nbas, T, seed=case)
    gb, gc, _ = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 1, 0, False, 1, 7.5)
    ob, oc, _ = oracle.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 1, 0, False, 1, 7.5)
    assert_same_functions(gb, gc, ob, oc, nbas, R, B)


@pytest.mark.gpu
@pytest.mark.parametrize("nbas,B,nals,eps", [([10] * 6, 40, 2, None), ([12, 7, 9], 18, 3, None), ([10] * 6, 12, 1, 3e-2),
                                             ([10] * 6, 12, 1, 1e-3)])
def test_one_cluster_against_the_grid_form(nbas, B, nals, eps, cuda_device):
    """Blocks of rank 16 run in one cluster; the same block stored at rank 17, every
    vector of rank 16, takes the grid form and fits the same terms."""
    R = 16
    rng = np.random.default_rng(5)
    if eps is None:
        Q, qc = rng.uniform(-0.5, 0.5, size=(B * R, sum(nbas))), rng.uniform(0.5, 1.0, B * R)
    else:
        Q, qc = close_terms(nbas, R, B, eps, 9)
    hl = H.random_hoplist(nbas, 3, seed=1)
    a = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, False, 1, 0.0)
    wide, wc = rng.uniform(-0.5, 0.5, size=(B, R + 1, sum(nbas))), np.zeros((B, R + 1))
    wide[:, :R], wc[:, :R] = Q.reshape(B, R, -1), qc.reshape(B, R)
    b = IT.intertwine(wide.reshape(B * (R + 1), -1), wc.reshape(-1), hl.nbas, R + 1, B, hl, np.zeros(B), 0, nals, False, 1,
                      0.0, ranks=[R] * B)
    assert not np.any(b[1].reshape(B, R + 1)[:, R])
    assert_same_functions(a[0], a[1], b[0], b[1], nbas, R, B, R + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n,R,B,nals", [(12, 1, 5, 1), (33, 3, 4, 2), (64, 17, 3, 1)])
def test_one_mode_block(n, R, B, nals, cuda_device):
    """With one mode a vector is one function, its normal equations are all ones (singular but
    for the penalty), and the stage is the plain Gram-Schmidt of the functions."""
    rng = np.random.default_rng(R)
    Q, qc = rng.uniform(-0.5, 0.5, size=(B * R, n)), rng.uniform(0.5, 1.0, B * R)
    A = rng.normal(size=(n, n))
    hl = H.build_hoplist([n], [(1.0, {0: A + A.T})])
    gb, gc, _ = IT.intertwine(Q, qc, hl.nbas, R, B, hl, np.zeros(B), 0, nals, False, 1, 0.0)
    f = np.einsum("vr,vrn->vn", qc.reshape(B, R), Q.reshape(B, R, n))
    g = np.einsum("vr,vrn->vn", gc.reshape(B, R), gb.reshape(B, R, n))
    q, r = np.linalg.qr(f.T)
    expected = (q * np.sign(np.diag(r))).T
    overlap = np.einsum("vn,vn->v", g, expected) / np.linalg.norm(g, axis=1)
    assert np.all(1 - overlap <= 1e-10)
