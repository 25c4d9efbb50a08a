"""The weight-gradient kernel with several work items a CTA: slots of the halo and
gradient rings that are used again, the gradient tiles kept twice, the count of tiles
carried from item to item, and items of unequal length in one CTA; against autograd."""
import numpy as np
import pytest

from oracle import closure_ref as cr
from simpletcsolver_b200.closure import LAYERS, _p

pytestmark = pytest.mark.gpu


# column tiles x chunks of planes: 64 x (7 of 5, 1 of 2), 128 x (3 of 4, 1 of 1) and
# 160 x (12, 11), all more than there are CTAs
@pytest.mark.parametrize("layer", range(4))
@pytest.mark.parametrize("grid", [(64, 128, 37), (64, 256, 13), (80, 256, 23)])
def test_weight_gradient_items(lib, grid, layer):
    import torch
    nx, ny, nz = grid
    cin, cp, cout, op = LAYERS[layer]
    gen = torch.Generator(device="cuda").manual_seed(11)
    x = torch.zeros(nz, ny, nx, cp, device="cuda")
    x[..., :cin] = torch.randn(nz, ny, nx, cin, generator=gen, device="cuda")
    g = torch.zeros(nz, ny, nx, op, device="cuda")
    g[..., :cout] = torch.randn(nz, ny, nx, cout, generator=gen, device="cuda")
    x, g = x.bfloat16(), g.bfloat16()
    w = torch.zeros(27, cout, cin, dtype=torch.float64, device="cuda", requires_grad=True)
    want, = torch.autograd.grad(cr.conv(x[..., :cin].double(), w), w, g[..., :cout].double())
    wb = g[..., :cout].double().sum((0, 1, 2))
    ws_bytes = lib.tcgpu_nn_wgrad_workspace(nx, ny, nz, op)
    ws = torch.empty(ws_bytes // 4, device="cuda").fill_(float("nan"))
    dw, db = torch.zeros(27, cout, cin, device="cuda"), torch.zeros(cout, device="cuda")
    torch.cuda.synchronize()
    assert lib.tcgpu_nn_conv3_wgrad(cp, op, cin, cout, nx, ny, nz, _p(x), _p(g), _p(dw), _p(db), 0.0, _p(ws), ws_bytes,
                                    None) == 0
    torch.cuda.synchronize()
    assert lib.tcgpu_nn_status(1) == 0
    # exact BF16 products, summed in FP32: n terms of unit variance, error about n 2^-24
    # of the terms' root sum of squares, sqrt(n) (a factor 8 over it); a plane that is
    # missed or counted twice changes the sums by some sqrt(nx ny)
    n = nx * ny * nz
    tol = 8 * n * 2.0 ** -24
    assert tol < 0.01 * (nx * ny) ** 0.5
    np.testing.assert_allclose(dw.cpu().double().numpy(), want.cpu().numpy(), rtol=0, atol=tol)
    np.testing.assert_allclose(db.cpu().double().numpy(), wb.cpu().numpy(), rtol=0, atol=tol)
