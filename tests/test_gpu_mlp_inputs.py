"""The warm-start network's backward pass on inputs that are not one contiguous BF16
block: rows further apart than they are long, through mlcp_mlp_step, and tensors of another
order, type or device, through Mlp.backward.  The reference is the same pass on a packed
copy: the values are the same, so the gradients are the same bits.
"""
import ctypes

import pytest
import torch

from mlcp_gb300 import _lib
from mlcp_gb300.mlp import Mlp, torch_stream


def network(rows, cuda_device):
    net = Mlp(64, 48, hidden=64, seed=3, device=cuda_device)
    g = torch.Generator().manual_seed(rows)
    X, _ = net.pad_inputs(torch.randn((rows, 64), generator=g))
    T = torch.randn((X.shape[0], net.out_p), generator=g).to(cuda_device)
    return net, X, T


def gradients(net):
    return [Ly[k].clone() for Ly in net.layers for k in ("gw", "gb")]


def step(net, backward, X, ldx, rows, *more):
    bufs = [net.status, X, net.H1, net.H1t, net.H2, net.H2t, net.Y]
    for Ly in net.layers:
        bufs += (Ly["wb"], Ly["b"])
    bufs += more
    t = (ctypes.c_void_p * len(bufs))(*[b.data_ptr() for b in bufs])
    dims = (ctypes.c_int * 7)(net.Y.shape[0], rows, net.in_p, net.h_p, net.out_p, net.out_dim, ldx)
    _lib.check(_lib.load().mlcp_mlp_step(backward, t, dims, torch_stream()))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,extra", [(100, 8), (200, 64), (128, 200)])
def test_row_stride_of_the_inputs(rows, extra, cuda_device):
    net, X, T = network(rows, cuda_device)
    net.forward(X, rows)
    net.backward(X, rows, T)
    expected = gradients(net)
    wide = torch.full((X.shape[0], net.in_p + extra), 7.0, dtype=torch.bfloat16, device=cuda_device)
    wide[:, :net.in_p] = X
    more = [T, net.loss, net.Xt, net.dY, net.dYt, net.dZ2, net.dZ2t, net.dZ1, net.dZ1t]
    for Ly in net.layers:
        Ly["gw"].zero_()
        more += (Ly["wt"], Ly["gw"], Ly["gb"])
    step(net, 0, wide, wide.shape[1], rows)
    step(net, 1, wide, wide.shape[1], rows, *more)
    for a, b in zip(expected, gradients(net)):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["columns first", "FP32", "every other row", "host"])
def test_backward_takes_any_tensor_of_the_inputs(form, cuda_device):
    rows = 100
    net, X, T = network(rows, cuda_device)
    net.forward(X, rows)
    net.backward(X, rows, T)
    expected = gradients(net)
    other = {"columns first": lambda: X.t().contiguous().t(), "FP32": X.float, "host": X.cpu,
             "every other row": lambda: X.repeat_interleave(2, 0)[::2]}[form]()
    assert other.shape == X.shape
    net.backward(other, rows, T)
    for a, b in zip(expected, gradients(net)):
        assert torch.equal(a, b)
