"""Tensor-core weight gradients of 16-bit operands over their channel counts (multiples of 8: padded
offset slots, columns past c_out), in index order and over a row order, with the data gradient and
the fused bias and ReLU gradient, against FP64 on the same operands.

Tolerances (relative L2): FP32 accumulation (2e-5) and one rounding of the result to the data type
(eps / 2); the fused-ReLU gradients see the layer's own rounded output as their mask, as the oracle
does here."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def f64(t):
    return t.detach().double().cpu().numpy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cin,cout,ks,n", [(8, 8, 3, 300), (16, 24, 3, 5003), (96, 40, 2, 5003), (64, 64, 3, 18000),
                                           (128, 256, 3, 1000), (40, 136, 3, 17003), (32, 96, 5, 2000)])
@pytest.mark.parametrize("transposed", [False, True])
def test_gradients(cuda_device, dtype, cin, cout, ks, n, transposed):
    import fvdb

    st = ks if ks == 2 else 1
    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(n, 36, n)).to(cuda_device))
    pack, tgt = grid.sparse_conv_kernel_map(ks, st)
    n_in, n_out = (tgt.total_voxels, grid.total_voxels) if transposed else (grid.total_voxels, tgt.total_voxels)
    g = torch.Generator().manual_seed(cin + cout)
    x = torch.randn(n_in, cin, generator=g).to(cuda_device, dtype).requires_grad_(True)
    shape = ((cin, cout) if transposed else (cout, cin)) + (ks,) * 3
    w = (torch.randn(shape, generator=g) / (cin * ks**3) ** 0.5).to(cuda_device, dtype).requires_grad_(True)
    b = (torch.randn(cout, generator=g) * 0.1).to(cuda_device, dtype).requires_grad_(True)
    dy = torch.randn(n_out, cout, generator=g).to(cuda_device, dtype)
    src, t = grid.ijk.jdata.cpu().numpy(), tgt.ijk.jdata.cpu().numpy()
    kmap = orc.kernel_map(src, np.array([0, src.shape[0]]), t, np.array([0, t.shape[0]]), ks, st)
    lim = torch.finfo(dtype).eps / 2 + 2e-5
    for _ in range(2):  # the second pass finds the row order built where the first did not
        y = pack._conv_with_bias(x, w, b, transposed, None, True).jdata
        dx, dw, db = torch.autograd.grad(y, [x, w, b], dy)
        m = f64(dy) * (f64(y) > 0)
        dx_ref, dw_ref = orc.conv_backward_f64(f64(x), f64(w), kmap, m, transposed=transposed, n_src=grid.total_voxels)
        assert dw.shape == w.shape and dw.dtype == dx.dtype == db.dtype == dtype
        assert rel(f64(dw), dw_ref) <= lim
        assert rel(f64(dx), dx_ref) <= lim
        assert rel(f64(db), m.sum(0)) <= lim
    torch.cuda.synchronize()
    fvdb._lib.load().check_device_errors(cuda_device)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,c", [(1, 1), (63, 5), (1000, 64), (257, 2056), (300, 1030)])
def test_bias_and_relu_gradient(cuda_device, dtype, n, c):
    """The masked gradient equals dy * (y > 0) bit for bit (a NaN or infinity under the mask
    included), with and without the ReLU; its column sums agree to FP32 accumulation."""
    import fvdb

    g = torch.Generator().manual_seed(n + c)
    dy = torch.randn(n, c, generator=g).to(cuda_device, dtype)
    y = torch.randn(n, c, generator=g).to(cuda_device, dtype)
    C = fvdb._lib.load()
    out, db = C.bias_relu_backward(dy, y, True)
    want = dy * (y > 0)
    assert torch.equal(out, want)
    tol = 1e-12 if dtype == torch.float64 else 1e-5
    scale = dy.double().abs().sum(0).clamp(min=1e-30)
    assert (((db.double() - want.double().sum(0)).abs() / scale) <= tol).all()
    same, db = C.bias_relu_backward(dy, None, True)
    assert torch.equal(same, dy) and (((db.double() - dy.double().sum(0)).abs() / scale) <= tol).all()
    dy[0, 0], y[0, 0] = float("inf"), -1.0
    out, _ = C.bias_relu_backward(dy, y, False)
    assert out[0, 0].isnan()
