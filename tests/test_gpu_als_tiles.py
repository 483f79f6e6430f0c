"""The explicit-target ALS at the edges of its tiles: 127, 128 and 129 target terms of
a CTA (a partial, a full, a full and a partial tile of 128), one tile with an idle
last warp (the normal equations are then inverted during the contraction) and
as many tiles as warps of a group, F ranks that fill their groups of four or not,
clusters of one, two and sixteen CTAs.  The checks and tolerances of one
sweep are those of test_gpu_als.py.
"""
import pytest

from mlcp_gb300 import workloads
from test_gpu_als import SWEEP_RES_TOL, SWEEP_VEC_TOL, compare, run_gpu

CASES = [  # vectors, modes, basis, rank, target terms
    (152, 3, 6, 4, 127),
    (152, 3, 6, 5, 128),
    (152, 3, 6, 5, 129),
    (76, 4, 5, 7, 512),
    (76, 3, 12, 20, 513),
    (1, 5, 9, 16, 40),
    (1, 4, 20, 16, 2100),
    (2, 3, 17, 33, 700),
    (9, 3, 12, 64, 300),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_sweep_at_tile_edges(case, cuda_device):
    nvec, D, n, rF, rG = case
    batch = workloads.als_batch(nvec, D, n, rF, rG, seed=rG)
    coef, base, status = run_gpu(batch, 1, cuda_device)
    assert not status.any()
    compare(batch, coef, base, 1, SWEEP_RES_TOL, SWEEP_VEC_TOL)
