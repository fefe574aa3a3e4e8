"""The surrogate's convolution and weight-gradient forms by row length, where
one gives way to another and where their tiles end: rows that divide a tile
(whole-row form), rows of whole tiles (ring form) and others (gather form);
rows of whole groups of 16 voxels, in one, two and three segments of 64 (the
gradient by lines), and others (the transposing gradient)."""
import numpy as np
import pytest

from swap_gb300 import abi
from test_gpu_surrogate import conv3_ref

pytestmark = pytest.mark.gpu

SHAPES = [(1, 128, 1), (2, 32, 2), (16, 8, 3), (32, 4, 5), (64, 3, 2), (64, 1, 2), (48, 8, 1), (80, 8, 2), (24, 16, 1),
          (144, 8, 1)]


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 16), (32, 32)])
@pytest.mark.parametrize("dims", SHAPES)
def test_conv3_by_row_length(dims, cin, cout):
    # FP32 accumulation of exact BF16 products, as in test_gpu_surrogate.py
    import torch

    V = dims[0] * dims[1] * dims[2]
    g = torch.Generator().manual_seed(V + cin)
    X = torch.randn(V, cin, generator=g).to(torch.bfloat16)
    W = (0.1 * torch.randn(27, cout, cin, generator=g)).to(torch.bfloat16)
    b = torch.randn(cout, generator=g).float()
    want = conv3_ref(X, W, b, dims) if min(dims) > 1 else _conv3_roll(X, W, b, dims)
    Yf = torch.zeros(V, cout, device="cuda")
    dX, dW, db = X.cuda(), W.cuda(), b.cuda()
    r = abi.load().swap_conv3_check(*dims, cin, cout, dX.data_ptr(), dW.data_ptr(), db.data_ptr(), None,
                                    Yf.data_ptr(), 0)
    assert r == 0
    assert (Yf.cpu().double() - want).abs().max().item() / want.abs().max().item() < 1e-5


def _conv3_roll(X, W, b, dims):
    """conv3_ref for axes of one voxel, which circular padding does not take."""
    import torch

    nx, ny, nz = dims
    f = X.double().reshape(nz, ny, nx, -1)
    y = b.double().expand(nx * ny * nz, -1)
    for t in range(27):
        sh = (-(t // 9 - 1), -(t // 3 % 3 - 1), -(t % 3 - 1))
        y = y + torch.roll(f, sh, (0, 1, 2)).reshape(nx * ny * nz, -1) @ W[t].double().T
    return y


@pytest.mark.parametrize("dims", [(16, 8, 1), (48, 8, 1), (64, 3, 2), (80, 8, 2), (144, 8, 1), (256, 2, 3)])
def test_weight_gradient_by_lines(dims):
    """Against the CUDA-core sums of the same BF16 values: the same sums in
    another order (test_gpu_surrogate.py's bar)."""
    import torch

    from swap_gb300.hybrid import Surrogate

    V = dims[0] * dims[1] * dims[2]
    net = Surrogate(seed=7)
    net.norm(np.full(Surrogate.NIN, 0.1), np.full(Surrogate.NIN, 1.5), np.zeros(3), np.ones(3))
    g = torch.Generator().manual_seed(V)
    vin = torch.randn(V, Surrogate.NIN, generator=g).cuda()
    tgt = torch.randn(V, 3, generator=g).cuda()
    _, tc = net.grads(dims, vin.data_ptr(), tgt.data_ptr())
    net.set_weight_grad_cores(True)
    _, cc = net.grads(dims, vin.data_ptr(), tgt.data_ptr())
    for l in range(len(net.layers)):
        for a, b in zip(tc[l], cc[l]):
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b), l
    net.close()
