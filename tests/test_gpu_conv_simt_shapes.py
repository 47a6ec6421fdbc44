"""The CUDA-core convolution and weight gradient (FP32, FP64) over their channel tiles and vector
widths: 32- and 64-wide tiles and remainders, odd channel counts (element loads), FP32 halo weight
gradients over the map; against FP64 (relative L2 2e-6: FP32 accumulation; 1e-13 in FP64)."""

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


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-13)])
@pytest.mark.parametrize("cin,cout,n", [(32, 64, 3000), (64, 32, 777), (3, 5, 1000), (33, 66, 500), (100, 36, 400), (16, 16, 40),
                                        (24, 200, 600)])
def test_forward_and_gradients(cuda_device, dtype, tol, cin, cout, n):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(n, 18, n)).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    g = torch.Generator().manual_seed(cin + cout)
    x = torch.randn(grid.total_voxels, cin, generator=g, dtype=dtype).to(cuda_device).requires_grad_(True)
    w = (torch.randn(cout, cin, 3, 3, 3, generator=g, dtype=dtype) / (27 * cin) ** 0.5).to(cuda_device).requires_grad_(True)
    dy = torch.randn(grid.total_voxels, cout, generator=g, dtype=dtype).to(cuda_device)
    ijk = grid.ijk.jdata.cpu().numpy()
    kmap = orc.kernel_map(ijk, np.array([0, n]), ijk, np.array([0, n]), 3, 1)
    y_ref = orc.conv_forward_f64(f64(x), f64(w), kmap)
    dx_ref, dw_ref = orc.conv_backward_f64(f64(x), f64(w), kmap, f64(dy))
    for conv in (lambda: pack.sparse_conv_3d(x, w).jdata, lambda: grid.sparse_conv_halo(grid.jagged_like(x), w).jdata):
        y = conv()
        dx, dw = torch.autograd.grad(y, [x, w], dy)
        assert rel(f64(y), y_ref) <= tol
        assert rel(f64(dx), dx_ref) <= tol
        assert rel(f64(dw), dw_ref) <= tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("cin,cout,n", [(8, 16, 900), (64, 32, 70000), (32, 64, 500), (3, 5, 300), (100, 36, 300)])
def test_bias_and_relu(cuda_device, dtype, cin, cout, n):
    """Bias and ReLU with the contraction's stores (short rows, narrow, wide and element-wise tiles, row
    order) equal the separate additions and clamps, bit for bit, NaN included."""
    import fvdb
    from fvdb import _lib

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(n, 64, n)).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    g = torch.Generator().manual_seed(cin + cout)
    x = torch.randn(grid.total_voxels, cin, generator=g, dtype=dtype).to(cuda_device)
    x[5] = float("nan")
    w = (torch.randn(cout, cin, 3, 3, 3, generator=g, dtype=dtype) / (27 * cin) ** 0.5).to(cuda_device)
    bias = torch.randn(cout, generator=g, dtype=dtype).to(cuda_device)
    conv = _lib.load().conv_forward
    y = conv(x, w, pack._impl, False)[0]
    bits = torch.int32 if dtype == torch.float32 else torch.int64
    for b, relu in ((bias, False), (bias, True), (None, True)):
        got = conv(x, w, pack._impl, False, b, relu)[0]
        ref = y if b is None else y + b
        ref = torch.relu(ref) if relu else ref
        nan = torch.isnan(ref)
        assert torch.equal(torch.isnan(got), nan)
        assert torch.equal(got[~nan].view(bits), ref[~nan].view(bits))
