"""Tensor-core convolutions of 16-bit features whose rows do not tile 128 bytes (channel counts that
are multiples of 8 only), in FP16 and BF16: forward with bias and ReLU, strided, transposed, the
data gradient and a reused map, against FP64 on the same operands.

Tolerance (relative L2): one rounding of the output (the type's unit roundoff, eps / 2) on FP32
accumulation of at most 27 x 136 products (2e-5)."""

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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("cin,cout,ks,st,transposed", [
    (8, 16, 3, 1, False), (24, 40, 3, 1, False), (40, 24, 2, 2, False), (48, 72, 3, 1, False), (72, 33, 3, 1, False),
    (136, 96, 2, 2, True), (16, 256, 3, 1, False), (56, 8, 2, 2, True), (64, 64, 3, 1, False),
])
def test_forward_and_data_gradient(cuda_device, dtype, cin, cout, ks, st, transposed):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(5003, 28, cin + cout)).to(cuda_device))
    pack, tgt = grid.sparse_conv_kernel_map(ks, st)
    n_in, n_out = (tgt.total_voxels, grid.total_voxels) if transposed else (grid.total_voxels, tgt.total_voxels)
    g = torch.Generator().manual_seed(cin)
    x = torch.randn(n_in, cin, generator=g).to(cuda_device, dtype).requires_grad_(True)
    shape = ((cin, cout) if transposed else (cout, cin)) + (ks,) * 3
    w = (torch.randn(shape, generator=g) / (cin * ks**3) ** 0.5).to(cuda_device, dtype)
    b = (torch.randn(cout, generator=g) * 0.1).to(cuda_device, dtype)
    dy = torch.randn(n_out, cout, generator=g).to(cuda_device, dtype)
    src, t = grid.ijk.jdata.cpu().numpy(), tgt.ijk.jdata.cpu().numpy()
    kmap = orc.kernel_map(src, np.array([0, src.shape[0]]), t, np.array([0, t.shape[0]]), ks, st)
    ref = orc.conv_forward_f64(f64(x), f64(w), kmap, transposed=transposed, n_src=grid.total_voxels)
    dx_ref, _ = orc.conv_backward_f64(f64(x), f64(w), kmap, f64(dy), transposed=transposed, n_src=grid.total_voxels)
    lim = torch.finfo(dtype).eps / 2 + 2e-5
    for _ in range(2):  # the second pass runs over the map's row order
        y = pack._conv_with_bias(x, w, b, transposed).jdata
        yr = pack._conv_with_bias(x.detach(), w, b, transposed, None, True).jdata
        (dx,) = torch.autograd.grad(y, x, dy)
        assert y.dtype == dtype
        assert rel(f64(y), ref + f64(b)) <= lim
        assert torch.equal(yr, y.detach().clamp(min=0))
        assert rel(f64(dx), dx_ref) <= lim
    torch.cuda.synchronize()
    fvdb._lib.load().check_device_errors(cuda_device)
