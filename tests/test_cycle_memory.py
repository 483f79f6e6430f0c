"""Device memory of one cycle as intwdevicemem_ reports it (host code; no GPU needed).

A block of more vectors than the Rayleigh-Ritz stage takes (160) runs without that
stage, so it needs none of its workspace: 24 squares of the block (the rotations of 30
Jacobi sweeps and nine matrices) beside the squares that every block has: three for the
matrices, R for the weights, D R^2 for the overlaps of its terms and R for their target
weights.  The rest grows with the block itself.
"""
import ctypes
import re

import pytest

from mlcp_gb300 import _lib


def workspace_mb(capfd, rk, nbas, nbloc, terms):
    L = _lib.load()
    i = lambda x: ctypes.byref(ctypes.c_int(x))  # noqa: E731
    D = len(nbas)
    L.intwdevicemem_(i(rk), i(D), i(nbloc), i(terms * D), i(terms * D + 2 * D), i(10 ** 9), i(1), ctypes.byref(ctypes.c_bool(False)),
                     (ctypes.c_int * D)(*nbas))
    ctypes.CDLL(None).fflush(None)
    return float(re.search(r"workspace\s*:\s*([0-9.]+) MB", capfd.readouterr().out).group(1))


@pytest.mark.parametrize("rk,nbas,nbloc", [(1, [10, 10], 20000), (1, [10, 10, 10], 8000), (4, [6, 6, 6], 5000)])
def test_large_blocks_need_no_rayleigh_ritz_workspace(rk, nbas, nbloc, capfd):
    D = len(nbas)
    squares = 3 + 2 * rk + D * rk * rk
    assert workspace_mb(capfd, rk, nbas, nbloc, 5) < (squares + 2) * 8.0 * nbloc ** 2 / 2 ** 20


def test_long_operator_lists_do_not_multiply_the_workspace(capfd):
    """160 vectors of rank 30 on six modes of 48 functions with 20000 terms: the operator Grams
    of all vectors are 138 GB, h F of every mode 221 GB.  The vectors are independent, so no more
    than 16 GB of that is held at once; the overlaps of the block's terms take 1.1 GB."""
    assert workspace_mb(capfd, 30, [48] * 6, 160, 20000) < 20 * 1024
