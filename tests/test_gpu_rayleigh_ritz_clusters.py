"""The generalised eigensolver of the Rayleigh-Ritz step (gep.cu) on clusters of
levels split on several scales.

A mode with one function beside a mode of n functions makes the block of all product
functions a plain symmetric eigenproblem of n levels with any spectrum: H is one dense
operator Q diag(levels) Q^T, and the two-mode reduction of the vectors (rank 1) adds no
error.  Tolerance: FP64 eigenpairs of a B x B matrix leave residuals and
orthogonality errors of a few B eps (here 5 B eps, relative to the largest level); nearly
degenerate levels are no exception.
"""
import numpy as np
import pytest

import oracle
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT
from test_gpu_rayleigh_ritz import product_block

EPS = np.finfo(float).eps


def shells(sizes, split):
    return np.concatenate([(k + 3.0) * (1.0 + split * np.arange(n)) for k, n in enumerate(sizes)])


def several_scales(smallest, count, size, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([(k + 3.0) * (1.0 + np.concatenate([[0.0], np.cumsum(10.0 ** rng.uniform(smallest, -3, size - 1))]))
                           for k in range(count)])


SPECTRA = {
    "shells_1e-6": shells((1, 6, 21, 12), 1e-6),
    "shells_1e-8": shells((1, 6, 21, 12), 1e-8),
    "shells_1e-10": shells((1, 6, 21, 12), 1e-10),
    "shells_1e-12": shells((1, 6, 21, 12), 1e-12),
    "shells_equal": shells((1, 6, 21, 12), 0.0),
    "scales_1e-8": several_scales(-8, 8, 8, 2),
    "scales_1e-11": several_scales(-11, 8, 8, 3),
    "scales_1e-14": several_scales(-14, 7, 9, 4),
    "geometric": np.logspace(-12, 0, 61),
    "cluster_at_zero": np.concatenate([np.linspace(-5, 5, 30), 1e-9 * np.arange(-8, 9)]),
    "small_block": 3.0 + 1e-10 * np.arange(7.0),
}


def rotated(levels, seed):
    q, _ = np.linalg.qr(np.random.default_rng(seed).normal(size=(len(levels), len(levels))))
    m = (q * levels) @ q.T
    return 0.5 * (m + m.T)


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SPECTRA))
def test_clustered_levels(name, cuda_device):
    levels = SPECTRA[name]
    B = len(levels)
    M = rotated(levels, B)
    hl = H.build_hoplist([1, B], [(1.0, {1: M})])
    base, coef = product_block(1, B, 1)
    gb, gc, ge = IT.diagonalize(base, coef, hl.nbas, 1, B, hl, 0)
    V = (gb[:, 0] * gc)[:, None] * gb[:, 1:]
    scale, tol = np.abs(levels).max(), 5 * B * EPS
    exact = np.linalg.eigvalsh(M)
    assert np.all(np.diff(ge) >= 0)
    assert np.abs(ge - exact).max() <= tol * scale
    assert np.abs(V @ M - ge[:, None] * V).max() <= tol * scale
    assert np.abs(V @ V.T - np.eye(B)).max() <= tol


@pytest.mark.gpu
@pytest.mark.parametrize("n1,n2,split", [(12, 12, 1e-7), (10, 16, 1e-9), (9, 11, 1e-5)])
def test_clustered_levels_of_two_modes(n1, n2, split, cuda_device):
    """Sums of two ladders whose spacings differ by `split`, and a weak coupling.  The
    vectors pass the two-mode reduction, so they are held to its bound (2e-11, as in
    test_gpu_rayleigh_ritz.py); the eigenvalues to the eigensolver's."""
    a, b = rotated(1.0 + np.arange(n1), 1), rotated((1.0 + split) * (1.0 + np.arange(n2)), 2)
    hl = H.build_hoplist([n1, n2], [(1.0, {0: a}), (1.0, {1: b}), (split, {0: rotated(np.linspace(-1, 1, n1), 3),
                                                                          1: rotated(np.linspace(-1, 1, n2), 4)})])
    B, rk = n1 * n2, min(n1, n2)
    base, coef = product_block(n1, n2, rk)
    gb, gc, ge = IT.diagonalize(base, coef, hl.nbas, rk, B, hl, 0)
    Hd = H.dense_hamiltonian(hl)
    exact = np.linalg.eigvalsh(Hd)
    scale = np.abs(exact).max()
    V = np.array([oracle.cp_dense(gb[v * rk:(v + 1) * rk], gc[v * rk:(v + 1) * rk], hl.nbas) for v in range(B)]).reshape(B, -1)
    assert np.abs(ge - exact).max() <= 5 * B * EPS * scale
    assert np.abs(V @ Hd - ge[:, None] * V).max() <= 2e-11 * scale
    assert np.abs(V @ V.T - np.eye(B)).max() <= 2e-11
