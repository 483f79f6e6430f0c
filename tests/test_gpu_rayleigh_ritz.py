"""The generalised eigensolver of the Rayleigh-Ritz step (gep.cu) through
diagonalizecpp_ on two-mode nodes whose block is every product function, so
that the answer is the node's exact spectrum and its vectors can be held to
H v = lambda v.

The sizes are the edges of its phases: one CTA up to 8 vectors, phase by
phase above; even and odd blocks (the round-robin schedule pads odd ones);
blocks that are and are not multiples of its tiles (8) and warps (32); the
largest (160).  The spectra are a force field's (separated), two equal
oscillators' (every sum of unlike levels doubly degenerate) and the same with
a coupling of 1e-9 (levels closer than the FP32 stage resolves).

Tolerance: FP64 eigenpairs of a B x B pencil leave residuals and
orthogonality errors of a few B eps (160 x 2.2e-16 = 3.5e-14); the vectors
come back as singular triplets, exact to 1e-12 (the reduction's own bound),
whose cut at 1e-12 s_1 may drop up to n such terms: 2e-11 relative.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT


def product_block(n1, n2, rk):
    base, coef = np.zeros((n1 * n2 * rk, n1 + n2)), np.zeros(n1 * n2 * rk)
    for a in range(n1):
        for b in range(n2):
            base[(a * n2 + b) * rk, [a, n1 + b]] = 1.0
            coef[(a * n2 + b) * rk] = 1.0
    return base, coef


def operators(kind, n1, n2):
    if kind == "field":
        return H.synthetic_qff(2, [n1, n2], 11)
    n = [n1, n2]
    terms = [(1.0, {d: 0.5 * (H.ho_p2(n[d]) + H.ho_q_power(n[d], 2))}) for d in range(2)]
    if kind == "close":
        terms.append((1e-9, {0: H.ho_q_power(n1, 1), 1: H.ho_q_power(n2, 1)}))
    return H.build_hoplist(n, terms)


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2", [(2, 1), (2, 2), (1, 8), (3, 3), (3, 5), (4, 4), (1, 17), (5, 5), (4, 8), (3, 11), (8, 8),
                                   (5, 13), (9, 11), (11, 13), (12, 12), (10, 16)])
@pytest.mark.parametrize("kind", ["field", "equal", "close"])
def test_product_block_gives_the_exact_spectrum(kind, n1, n2, cuda_device):
    hl = operators(kind, n1, n2)
    Hd = H.dense_hamiltonian(hl)
    B, rk = n1 * n2, min(n1, n2)
    base, coef = product_block(n1, n2, rk)
    gb, gc, ge = IT.diagonalize(base, coef, hl.nbas, rk, B, hl, 0)
    exact = np.linalg.eigvalsh(Hd)
    scale = np.abs(exact).max()
    assert np.all(np.diff(ge) >= 0)
    assert np.abs(ge - exact).max() <= 1e-13 * scale
    V = np.array([oracle.cp_dense(gb[v * rk:(v + 1) * rk], gc[v * rk:(v + 1) * rk], hl.nbas) for v in range(B)])
    V = V.reshape(B, -1)
    assert np.abs(V @ Hd - ge[:, None] * V).max() <= 2e-11 * scale
    assert np.abs(V @ V.T - np.eye(B)).max() <= 2e-11
