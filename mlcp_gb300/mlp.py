"""Three-layer MLP of the learned ALS warm start, trained and run by the
library's own kernels (``csrc/mlp.cu``): tcgen05 BF16 GEMMs with FP32
accumulation, ReLU, mean-squared-error loss, Adam on FP32 master weights.

Shapes (every GEMM dimension padded as the kernels need): inputs
``in_dim`` -> ``hidden`` -> ``hidden`` -> ``out_dim``.  Rows (samples),
hidden and output widths are padded to multiples of 128 (they are the M of
some GEMM), the input width to a multiple of 64; padding rows and columns
are zero and masked out of the loss.

Data layout: BF16 activations row-major [rows][width]; each layer also keeps
the transposed copy [width][rows] that its weight-gradient GEMM reads, and
each weight matrix [out][in] its transposed BF16 copy [in][out] that the
input-gradient GEMM reads.  Torch allocates the device buffers; every
computation is a call into libmlcp_gb300.
"""
from __future__ import annotations

import ctypes

import numpy as np

from . import _lib


def _pad(x: int, m: int) -> int:
    return (x + m - 1) // m * m


def torch_stream():
    """Handle of torch's current stream for the library calls, so that they
    order with the torch operations that fill and read the buffers (the
    legacy default stream is passed as its special handle 1, since NULL
    selects the library's own stream)."""
    import torch
    return torch.cuda.current_stream().cuda_stream or 1


class Mlp:
    """MLP with device-resident parameters.  ``params()`` returns FP32 master
    copies (W1, b1, W2, b2, W3, b3) as numpy arrays of the logical shapes."""

    def __init__(self, in_dim: int, out_dim: int, hidden: int = 256, seed: int = 0, device=None):
        import torch
        self.torch = torch
        self.dev = device or torch.device("cuda", torch.cuda.current_device())
        self.in_dim, self.out_dim, self.hidden = in_dim, out_dim, hidden
        self.in_p = _pad(in_dim, 64)
        self.h_p = _pad(hidden, 128)
        self.out_p = _pad(out_dim, 128)
        rng = np.random.default_rng(seed)
        dims = [(self.h_p, self.in_p, hidden, in_dim), (self.h_p, self.h_p, hidden, hidden),
                (self.out_p, self.h_p, out_dim, hidden)]
        self.layers = []
        for (rp, cp, r, c) in dims:
            w = np.zeros((rp, cp), dtype=np.float32)
            w[:r, :c] = rng.uniform(-1.0, 1.0, size=(r, c)) * np.sqrt(3.0 / c)
            L = {"rows": rp, "cols": cp,
                 "w": torch.from_numpy(w).to(self.dev), "b": torch.zeros(rp, dtype=torch.float32, device=self.dev)}
            for k in ("mw", "vw"):
                L[k] = torch.zeros_like(L["w"])
            for k in ("mb", "vb"):
                L[k] = torch.zeros_like(L["b"])
            L["gw"] = torch.zeros_like(L["w"])
            L["gb"] = torch.zeros_like(L["b"])
            L["wb"] = L["w"].to(torch.bfloat16).contiguous()
            L["wt"] = L["w"].t().contiguous().to(torch.bfloat16)
            self.layers.append(L)
        self.step_no = 0
        self.status = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self._rows = 0

    # -- buffers for a number of padded rows --
    def _buffers(self, rows_p: int):
        if rows_p == self._rows:
            return
        t = self.torch
        bf = t.bfloat16
        z = lambda r, c, dt=bf: t.zeros((r, c), dtype=dt, device=self.dev)  # noqa: E731
        self.H1, self.H1t = z(rows_p, self.h_p), z(self.h_p, rows_p)
        self.H2, self.H2t = z(rows_p, self.h_p), z(self.h_p, rows_p)
        self.Y = z(rows_p, self.out_p, t.float32)
        self.dY, self.dYt = z(rows_p, self.out_p), z(self.out_p, rows_p)
        self.dZ2, self.dZ2t = z(rows_p, self.h_p), z(self.h_p, rows_p)
        self.dZ1, self.dZ1t = z(rows_p, self.h_p), z(self.h_p, rows_p)
        self.Xt = z(self.in_p, rows_p)
        self.loss = t.zeros(1, dtype=t.float32, device=self.dev)
        self._rows = rows_p

    def _step(self, backward: bool, Xp, rows: int, *more):
        """One library call for all launches of a pass: the buffers' addresses of
        this call, in the order of mlcp_mlp_step."""
        bufs = [self.status, Xp, self.H1, self.H1t, self.H2, self.H2t, self.Y]
        for Ly in self.layers:
            bufs += (Ly["wb"], Ly["b"])
        bufs += more
        t = (ctypes.c_void_p * len(bufs))(*[b.data_ptr() for b in bufs])
        dims = (ctypes.c_int * 7)(Xp.shape[0], rows, self.in_p, self.h_p, self.out_p, self.out_dim, Xp.shape[1])
        _lib.check(_lib.load().mlcp_mlp_step(int(backward), t, dims, torch_stream()))

    def pad_inputs(self, X):
        """BF16 [rows_p][in_p] copy of X (rows x in_dim, any float dtype)."""
        t = self.torch
        rows = X.shape[0]
        rows_p = _pad(max(rows, 1), 128)
        Xp = t.zeros((rows_p, self.in_p), dtype=t.bfloat16, device=self.dev)
        Xp[:rows, :X.shape[1]] = X.to(t.bfloat16)
        return Xp, rows

    def forward(self, Xp, rows: int):
        """Xp: BF16 [rows_p][in_p] (pad_inputs).  Returns Y FP32 [rows_p][out_p]."""
        self._buffers(Xp.shape[0])
        self._step(False, Xp, rows)
        return self.Y

    def backward(self, Xp, rows: int, T):
        """Gradients of the mean squared error of the last forward against T
        (FP32 [rows_p][out_p]; columns >= out_dim ignored) into each layer's
        gw/gb.  Returns the loss (device scalar)."""
        if tuple(Xp.shape) != (self._rows, self.in_p):
            raise RuntimeError(f"inputs of shape {tuple(Xp.shape)}, the last forward's were {(self._rows, self.in_p)}")
        if Xp.dtype != self.Xt.dtype or Xp.device != self.Xt.device or not Xp.is_contiguous():
            Xp = Xp.to(device=self.dev, dtype=self.Xt.dtype).contiguous()
        more = [T, self.loss, self.Xt, self.dY, self.dYt, self.dZ2, self.dZ2t, self.dZ1, self.dZ1t]
        for Ly in self.layers:
            more += (Ly["wt"], Ly["gw"], Ly["gb"])
        self._step(True, Xp, rows, *more)
        return self.loss

    def adam(self, lr: float = 1e-3, b1: float = 0.9, b2: float = 0.999, eps: float = 1e-8):
        self.step_no += 1
        t, dims = [], []
        for Ly in self.layers:
            t += [Ly[k].data_ptr() for k in ("w", "gw", "mw", "vw", "wb", "wt")]
            t += [Ly[k].data_ptr() for k in ("b", "gb", "mb", "vb")] + [None, None]
            dims += (Ly["rows"], Ly["cols"], 1, Ly["rows"])
        _lib.check(_lib.load().mlcp_mlp_adam_layers(6, (ctypes.c_void_p * 36)(*t), (ctypes.c_int * 12)(*dims), lr, b1, b2,
                                                    eps, self.step_no, torch_stream()))

    def check_status(self):
        if int(self.status.item()) != 0:
            raise _lib.MlcpError("mlp gemm: an internal wait timed out")

    def params(self):
        out = []
        for Ly, (r, c) in zip(self.layers, [(self.hidden, self.in_dim), (self.hidden, self.hidden),
                                            (self.out_dim, self.hidden)]):
            out.append(Ly["w"][:r, :c].cpu().numpy().astype(np.float64))
            out.append(Ly["b"][:r].cpu().numpy().astype(np.float64))
        return out

    def grads(self):
        out = []
        for Ly, (r, c) in zip(self.layers, [(self.hidden, self.in_dim), (self.hidden, self.hidden),
                                            (self.out_dim, self.hidden)]):
            out.append(Ly["gw"][:r, :c].cpu().numpy().astype(np.float64))
            out.append(Ly["gb"][:r].cpu().numpy().astype(np.float64))
        return out
