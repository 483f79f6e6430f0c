"""The passes of the warm-start network that run from one library call each
(mlcp_mlp_step, mlcp_mlp_adam_layers) against the same passes as single calls of
mlcp_mlp_gemm, mlcp_mlp_loss, mlcp_mlp_colsum and mlcp_mlp_adam: the kernels and
their order within every sum are the same, so all results are the same bits, but
the loss, whose tiles' parts meet by atomics (2e3 parts at most, so within 2e3 2^-24).
Widths that fill their padding and that do not, one and several row blocks.
"""
import ctypes

import pytest
import torch

from mlcp_gb300 import _lib
from mlcp_gb300.mlp import Mlp, torch_stream

CASES = [(64, 128, 128, 128), (100, 37, 256, 200), (5, 130, 64, 640), (576, 256, 256, 769)]  # in, out, hidden, rows


def gemm(A, B, M, N, K, status, bias=None, act=0, mask=None, C=None, Cb=None, Ct=None, valid_m=None):
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    ld = lambda t: 0 if t is None else t.shape[1]  # noqa: E731
    _lib.check(_lib.load().mlcp_mlp_gemm(p(A), p(B), M, N, K, A.shape[1], B.shape[1], p(bias), act, p(mask), ld(mask), p(C),
                                         ld(C), p(Cb), ld(Cb), p(Ct), ld(Ct), M if valid_m is None else valid_m,
                                         p(status), torch_stream()))


def step_by_calls(n, X, rows, T, lr):
    L, M, h, o = _lib.load(), X.shape[0], n.h_p, n.out_p
    a, b, c = n.layers
    n._buffers(M)
    gemm(X, a["wb"], M, h, n.in_p, n.status, a["b"], 1, Cb=n.H1, Ct=n.H1t, valid_m=rows)
    gemm(n.H1, b["wb"], M, h, h, n.status, b["b"], 1, Cb=n.H2, Ct=n.H2t, valid_m=rows)
    gemm(n.H2, c["wb"], M, o, h, n.status, c["b"], 0, C=n.Y, valid_m=rows)
    n.loss.zero_()
    _lib.check(L.mlcp_mlp_loss(n.Y.data_ptr(), T.data_ptr(), rows, n.out_dim, o, M, n.dY.data_ptr(), n.dYt.data_ptr(),
                               n.loss.data_ptr(), torch_stream()))
    n.Xt.copy_(X.t())
    gemm(n.dYt, n.H2t, o, h, M, n.status, C=c["gw"])
    gemm(n.dY, c["wt"], M, h, o, n.status, act=2, mask=n.H2, Cb=n.dZ2, Ct=n.dZ2t, valid_m=rows)
    gemm(n.dZ2t, n.H1t, h, h, M, n.status, C=b["gw"])
    gemm(n.dZ2, b["wt"], M, h, h, n.status, act=2, mask=n.H1, Cb=n.dZ1, Ct=n.dZ1t, valid_m=rows)
    gemm(n.dZ1t, n.Xt, h, n.in_p, M, n.status, C=a["gw"])
    for G, Ly in ((n.dY, c), (n.dZ2, b), (n.dZ1, a)):
        _lib.check(L.mlcp_mlp_colsum(G.data_ptr(), M, G.shape[1], G.shape[1], Ly["gb"].data_ptr(), torch_stream()))
    n.step_no += 1
    f = ctypes.c_float
    for Ly in n.layers:
        for w, g, m, v, r, k, wb, wt in ((*(Ly[q].data_ptr() for q in ("w", "gw", "mw", "vw")), Ly["rows"], Ly["cols"],
                                          Ly["wb"].data_ptr(), Ly["wt"].data_ptr()),
                                         (*(Ly[q].data_ptr() for q in ("b", "gb", "mb", "vb")), 1, Ly["rows"], None, None)):
            _lib.check(L.mlcp_mlp_adam(w, g, m, v, r, k, f(lr), f(0.9), f(0.999), f(1e-8), n.step_no, wb, wt,
                                       torch_stream()))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_passes_match_single_calls(case, cuda_device):
    n_in, n_out, hidden, rows = case
    one, many = (Mlp(n_in, n_out, hidden=hidden, seed=4, device=cuda_device) for _ in range(2))
    g = torch.Generator().manual_seed(rows)
    X, _ = one.pad_inputs(torch.rand(rows, n_in, generator=g).to(cuda_device))
    T = torch.zeros(X.shape[0], one.out_p, device=cuda_device)
    T[:rows, :n_out] = torch.rand(rows, n_out, generator=g).to(cuda_device)
    for _ in range(2):
        one.forward(X, rows)
        loss = one.backward(X, rows, T)
        one.adam(lr=1e-3)
        step_by_calls(many, X, rows, T, 1e-3)
        torch.testing.assert_close(loss, many.loss, rtol=2e3 * 2.0 ** -24, atol=0)
        assert torch.equal(one.Y, many.Y)
        for a, b in zip(one.layers, many.layers):
            for k in ("gw", "gb", "w", "b", "mw", "vw", "mb", "vb", "wb", "wt"):
                assert torch.equal(a[k], b[k]), k
    one.check_status()


@pytest.mark.gpu
def test_backward_refuses_other_inputs(cuda_device):
    net = Mlp(20, 10, device=cuda_device)
    X, rows = net.pad_inputs(torch.ones(5, 20, device=cuda_device))
    net.forward(X, rows)
    with pytest.raises(RuntimeError):
        net.backward(torch.cat([X, X]), rows, torch.zeros(256, net.out_p, device=cuda_device))
