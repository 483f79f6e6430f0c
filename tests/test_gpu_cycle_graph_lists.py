"""The cycle's CUDA graph across operator lists of one shape: two lists that agree
in every total (modes, terms, basis functions, operators, the largest mode of
each) but spread them differently over the modes need different launches, as a mode tree
that solves node after node produces.  The same calls with the graph off are the
reference: the kernels are the same, so the results are the same bits.  Each list is
called twice and the lists alternate, so that a graph is captured, replayed and
replaced.
"""
import numpy as np
import pytest

from mlcp_gb300 import _lib
from mlcp_gb300 import hoplist as H
from mlcp_gb300 import intertwine as IT


def operator_counts(hl):
    """Distinct operators per mode, the identity among them."""
    op = np.asarray(hl.opid).reshape(-1, len(hl.nbas))
    counts = []
    for d, n in enumerate(int(x) for x in hl.nbas):
        eye = H.pack(np.eye(n))
        starts = {int(hl.mptr[o - 1]) - 1 for o in op[:, d]}
        counts.append(1 + sum(not np.array_equal(hl.mat[s:s + n * (n + 1) // 2], eye) for s in starts))
    return counts


def lists(kind):
    if kind == "operators":  # (24, 21, 18) and (24, 23, 16) distinct operators
        return [H.random_hoplist([12, 10, 11], 30, seed) for seed in (5, 30)]
    if kind == "bases":
        return [H.random_hoplist(nb, 24, 2, coupling=3) for nb in ([33, 9, 17], [17, 33, 9])]
    small = [H.random_hoplist(nb, 6, 2, coupling=3) for nb in ([7, 4, 6], [6, 7, 4])]  # one CTA per vector
    assert kind == "small"
    return small


@pytest.mark.gpu
@pytest.mark.parametrize("kind,rk,nbloc", [("operators", 24, 4), ("bases", 18, 4), ("bases", 33, 3), ("small", 4, 5)])
@pytest.mark.parametrize("update", [False, True])
def test_lists_of_one_shape_keep_their_own_launches(kind, rk, nbloc, update, cuda_device):
    two = lists(kind)
    a, b = (operator_counts(hl) for hl in two)
    assert (sum(a), max(a), two[0].nterms) == (sum(b), max(b), two[1].nterms)
    assert a != b or list(two[0].nbas) != list(two[1].nbas)
    assert sum(two[0].nbas) == sum(two[1].nbas) and max(two[0].nbas) == max(two[1].nbas)
    L = _lib.load()
    rng = np.random.default_rng(7)
    Q, c = rng.uniform(-0.5, 0.5, size=(rk * nbloc, int(sum(two[0].nbas)))), np.ones(rk * nbloc)
    out = {}
    for graph in (0, 1):
        L.mlcp_gb300_set_cycle_graph(graph)
        try:
            out[graph] = [IT.intertwine(Q, c, hl.nbas, rk, nbloc, hl, np.zeros(nbloc), 2, 1, update, 1, 3.0)
                          for hl in (two[0], two[0], two[1], two[1], two[0], two[0])]
        finally:
            L.mlcp_gb300_set_cycle_graph(1)
    for off, on in zip(out[0], out[1]):
        for x, y in zip(off, on):
            np.testing.assert_array_equal(x, y)
