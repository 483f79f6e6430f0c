"""The dense solves of up to 16 rows (dwsolve.cuh) on systems of growing condition, by a
small program around the header (dwsolve_check.cu): the corrected inverse, which the
Gram-Schmidt multiplies its right-hand sides by, against the refinement of every
right-hand side, which it replaced there.

Both correct the same FP32 inverse with residuals in double-word and promise 1e-10 of the
solution.  Over the conditions that such corrections reach, the corrected inverse is to
take as many systems as the refinement (their stop rules look at different norms, so not
every single one), and its largest error over the systems it takes is to be no more than
four times that of the refinement (of the double-word LDL^T where the refinement gives up)
plus a tenth of that promise.  Systems: symmetric positive definite with unit diagonal,
exact in double-word; solutions of order one; the exact ones by refinement in extended
precision.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mlcp_gb300", "csrc")
CONDITIONS = [1e1, 1e3, 1e4, 3e4, 1e5]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    from mlcp_gb300 import build
    if not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")):
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("dwsolve") / "dwsolve_check.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
                    "-shared", "-I", CSRC, os.path.join(HERE, "dwsolve_check.cu"), "-o", so], check=True)
    return ctypes.CDLL(so)


def double_word(x):
    hi = x.astype(np.float32)
    return hi.astype(float) + (x - hi).astype(np.float32).astype(float)


def systems(n, condition, spectrum, count, nrhs, seed):
    rng = np.random.default_rng(seed)
    A = np.empty((count, n, n))
    lam = np.logspace(0, -np.log10(condition), n) if spectrum == "spread" else np.r_[np.ones(n - 1), 1 / condition]
    for s in range(count):
        q, _ = np.linalg.qr(rng.normal(size=(n, n)))
        a = (q * lam) @ q.T
        d = 1 / np.sqrt(np.diag(a))
        A[s] = 0.5 * (a + a.T) * d[:, None] * d[None, :]
    A = double_word(A)
    B = double_word(np.einsum("sij,srj->sri", A, rng.normal(size=(count, nrhs, n))))
    X = np.zeros(B.shape, np.longdouble)
    for s in range(count):
        inv, a, b = np.linalg.inv(A[s]), A[s].astype(np.longdouble), B[s].T.astype(np.longdouble)
        x = np.zeros_like(b)
        for _ in range(8):
            x = x + (inv @ (b - a @ x).astype(float)).astype(np.longdouble)
        X[s] = x.T
    return A, B, X


def solve(library, A, B):
    count, nrhs, n = B.shape
    X, solved, cycles = np.zeros((count, 3, nrhs, n)), np.zeros((count, 3), np.int32), np.zeros((count, 3), np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert library.dwsolve_check(n, nrhs, count, p(A), p(B), p(X), p(solved), p(cycles)) == 0
    return X, solved > 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 8, 16])
@pytest.mark.parametrize("spectrum", ["spread", "one"])
def test_corrected_inverse_is_no_worse_than_refinement(n, spectrum, library, cuda_device):
    taken = np.zeros(2, int)
    for condition in CONDITIONS:
        A, B, exact = systems(n, condition, spectrum, 100, 10, 5)
        X, solved = solve(library, np.ascontiguousarray(A), np.ascontiguousarray(B))
        refined, inverse = solved[:, 0], solved[:, 1]
        taken += refined.sum(), inverse.sum()
        error = (np.abs(X - exact[:, None]).max(axis=(2, 3)) / np.abs(exact).max(axis=(1, 2))[:, None]).astype(float)
        before = np.where(refined, error[:, 0], error[:, 2])
        if inverse.any():
            assert error[inverse, 1].max() <= 4 * before[inverse].max() + 1e-11, condition
    assert taken[1] >= taken[0]
