"""The tile widths, operand ring and epilogue stores of the warm start's GEMM
(csrc/mlp.cu): one shape for each width that the launch rule picks (32 up to
256 columns, by how many tiles the shape makes), more K slices than ring
stages, a last tile of 16 columns, and outputs whose rows do not start on
16-byte boundaries (element-wise stores).  The bound is the existing GEMM
test's: 1e-5 of the row's largest |product| sum, FP32 accumulation over K;
the BF16 copies are the rounded FP32 outputs bit for bit.

The bias gradient, the loss and Adam at sizes around their 32-wide tiles,
against FP64: sums of up to 257 terms in FP32, 257 x 2^-24 < 2e-5 of the sum
of magnitudes.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as MO


def bf(t):
    import torch
    return t.to(torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(128, 48, 1024), (256, 272, 640), (2432, 512, 576), (4864, 512, 320),
                                   (9728, 512, 320)])
@pytest.mark.parametrize("pad", [0, 1])
def test_gemm_tiles(M, N, K, pad, cuda_device):
    import torch
    from mlcp_gb300 import _lib
    from mlcp_gb300.mlp import torch_stream
    g = torch.Generator().manual_seed(M + N + K)
    A, B = bf(torch.randn(M, K, generator=g)).to(cuda_device), bf(torch.randn(N, K, generator=g)).to(cuda_device)
    bias = torch.randn(N, generator=g).float().to(cuda_device)
    mask = bf(torch.randn(M, N + pad, generator=g)).to(cuda_device)
    C = torch.full((M, N + pad), 7.0, dtype=torch.float32, device=cuda_device)
    Cb = torch.full((M, N + pad), 7.0, dtype=torch.bfloat16, device=cuda_device)
    Ct = torch.full((N, M + pad), 7.0, dtype=torch.bfloat16, device=cuda_device)
    st = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _lib.check(_lib.load().mlcp_mlp_gemm(A.data_ptr(), B.data_ptr(), M, N, K, K, K, bias.data_ptr(), 2,
                                         mask.data_ptr(), N + pad, C.data_ptr(), N + pad, Cb.data_ptr(), N + pad,
                                         Ct.data_ptr(), M + pad, M - 3, st.data_ptr(), torch_stream()))
    torch.cuda.synchronize()
    assert int(st.item()) == 0
    a, b = A.double(), B.double()
    ref = torch.where(mask[:, :N].double() > 0, a @ b.T + bias.double(), 0.0)
    ref[M - 3:] = 0.0
    scale = a.abs() @ b.abs().T + 1.0
    got = C[:, :N]
    assert float(((got.double() - ref).abs() / scale).max()) <= 1e-5
    assert torch.equal(Cb[:, :N], got.to(torch.bfloat16))
    assert torch.equal(Ct[:, :M].T, Cb[:, :N])
    if pad:  # nothing written beside the outputs
        assert bool((C[:, N:] == 7.0).all()) and bool((Cb[:, N:] == 7.0).all()) and bool((Ct[:, M:] == 7.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (64, 32), (257, 65)])
def test_gradient_and_optimiser_tiles(rows, cols, cuda_device):
    import ctypes

    import torch
    from mlcp_gb300 import _lib
    from mlcp_gb300.mlp import torch_stream
    L = _lib.load()
    rng = np.random.default_rng(rows + cols)
    dev = lambda x, dt=torch.float32: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device, dt)  # noqa: E731
    G = MO.bf16(rng.normal(size=(rows, cols)))
    db = torch.full((cols + 1,), 7.0, device=cuda_device)
    Gd = dev(G, torch.bfloat16)
    _lib.check(L.mlcp_mlp_colsum(Gd.data_ptr(), rows, cols, cols, db.data_ptr(), torch_stream()))
    assert np.all(np.abs(db[:cols].cpu().numpy() - G.sum(0)) <= 2e-5 * np.abs(G).sum(0) + 1e-30)
    assert float(db[cols]) == 7.0
    # loss over all but the last row and column
    Y, T = rng.normal(size=(rows, cols)).astype(np.float32), rng.normal(size=(rows, cols)).astype(np.float32)
    m, n = max(rows - 1, 1), max(cols - 1, 1)
    dY = torch.zeros((rows, cols), dtype=torch.bfloat16, device=cuda_device)
    dYt = torch.zeros((cols, rows), dtype=torch.bfloat16, device=cuda_device)
    loss = torch.zeros(1, device=cuda_device)
    Yd, Td = dev(Y), dev(T)
    _lib.check(L.mlcp_mlp_loss(Yd.data_ptr(), Td.data_ptr(), m, n, cols, rows, dY.data_ptr(), dYt.data_ptr(),
                               loss.data_ptr(), torch_stream()))
    d = (Y - T).astype(np.float64)
    d[m:] = 0.0
    d[:, n:] = 0.0
    assert abs(float(loss) - (d ** 2).sum() / (m * n)) <= 2e-5 * (d ** 2).sum() / (m * n)
    got = dY.float().cpu().numpy()
    assert np.abs(got - 2 * d / (m * n)).max() <= 2 ** -8 * np.abs(2 * d / (m * n)).max()
    assert torch.equal(dYt.T, dY)
    # one Adam step (the second: bias corrections of both moments)
    w, g, m1, m2 = (rng.normal(size=(rows, cols)).astype(np.float32) for _ in range(4))
    m2 = np.abs(m2)
    wd, gd, ad, bd = dev(w), dev(g), dev(m1), dev(m2)
    wb = torch.zeros((rows, cols), dtype=torch.bfloat16, device=cuda_device)
    wt = torch.zeros((cols, rows), dtype=torch.bfloat16, device=cuda_device)
    f = ctypes.c_float
    _lib.check(L.mlcp_mlp_adam(wd.data_ptr(), gd.data_ptr(), ad.data_ptr(), bd.data_ptr(), rows, cols, f(1e-2), f(0.9),
                               f(0.999), f(1e-8), 2, wb.data_ptr(), wt.data_ptr(), torch_stream()))
    a = 0.9 * m1.astype(np.float64) + 0.1 * g
    b = 0.999 * m2.astype(np.float64) + 0.001 * g.astype(np.float64) ** 2
    ref = w - 1e-2 * (a / (1 - 0.9 ** 2)) / (np.sqrt(b / (1 - 0.999 ** 2)) + 1e-8)
    # FP32 throughout; 1 - 0.999^2 from FP32 powers loses three digits
    assert np.abs(wd.cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref - w).max() + 1e-6
    assert torch.equal(wb, wd.to(torch.bfloat16)) and torch.equal(wt.T, wb)
