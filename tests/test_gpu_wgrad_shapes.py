"""The weight-gradient kernel where its shares of planes are short or ragged: single
planes, segments that cross column tiles, fewer planes than CTAs, accumulation, and a
workspace that starts at an odd float; against autograd on the CPU."""
import ctypes as C

import numpy as np
import pytest

from oracle import closure_ref as cr
from simpletcsolver_b200.closure import LAYERS, _p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", range(4))
@pytest.mark.parametrize("grid", [(8, 16, 1), (8, 16, 2), (16, 16, 3), (24, 48, 5), (8, 32, 37), (40, 112, 6)])
def test_weight_gradient_shapes(lib, grid, layer):
    import torch
    nx, ny, nz = grid
    cin, cp, cout, op = LAYERS[layer]
    gen = torch.Generator().manual_seed(7)
    x = torch.zeros(nz, ny, nx, cp)
    x[..., :cin] = torch.randn(nz, ny, nx, cin, generator=gen)
    g = torch.zeros(nz, ny, nx, op)
    g[..., :cout] = torch.randn(nz, ny, nx, cout, generator=gen)
    x, g = x.bfloat16(), g.bfloat16()
    w = torch.zeros(27, cout, cin, dtype=torch.float64, requires_grad=True)
    y = cr.conv(x[..., :cin].double(), w)
    want, = torch.autograd.grad(y, w, g[..., :cout].double())
    wb = g[..., :cout].double().sum((0, 1, 2))
    ws_bytes = lib.tcgpu_nn_wgrad_workspace(nx, ny, nz, op)
    ws = torch.zeros(ws_bytes // 4 + 1, device="cuda")
    dw, db = torch.full((27, cout, cin), 3.0, device="cuda"), torch.full((cout,), -2.0, device="cuda")
    xd, gd = x.cuda().contiguous(), g.cuda().contiguous()
    for beta in (0.0, 1.0):
        assert lib.tcgpu_nn_conv3_wgrad(cp, op, cin, cout, nx, ny, nz, _p(xd), _p(gd), _p(dw), _p(db), beta,
                                        C.c_void_p(ws.data_ptr() + 4), ws_bytes, None) == 0
    torch.cuda.synchronize()
    assert lib.tcgpu_nn_status(1) == 0
    # exact BF16 products, summed in FP32: n terms of unit variance, error about
    # n 2^-24 of the terms' root sum of squares, sqrt(n) (a factor 8 over it)
    n = nx * ny * nz
    tol = 2 * 8 * n ** 0.5 * max(n ** 0.5, 8.0) * 2.0 ** -24
    np.testing.assert_allclose(dw.cpu().double().numpy(), 2 * want.numpy(), rtol=0, atol=tol)
    np.testing.assert_allclose(db.cpu().double().numpy(), 2 * wb.numpy(), rtol=0, atol=tol)
