"""Layers under torch.inference_mode, and what it leaves behind: the same results as without it, and
weights, grids and maps that serve calls with and without gradients afterwards."""

import pytest
import torch

from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu


def _grid(fvdb, dev, n=2000, extent=20, seed=2):
    return fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(n, extent, seed)).to(dev))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("transposed", [False, True])
def test_convolution(cuda_device, dtype, transposed):
    import fvdb

    grid = _grid(fvdb, cuda_device)
    g = torch.Generator().manual_seed(1)
    w = (torch.randn(24, 24, 3, 3, 3, generator=g) * 0.05).to(cuda_device, dtype).requires_grad_(True)
    x = torch.randn(grid.total_voxels, 24, generator=g).to(cuda_device, dtype)

    def conv():
        pack, _ = grid.sparse_conv_kernel_map(3, 1)
        return (pack.sparse_transpose_conv_3d if transposed else pack.sparse_conv_3d)(x, w).jdata

    with torch.inference_mode():
        a, b = conv(), conv()
    assert a.is_inference()
    with torch.no_grad():
        c = conv()
    assert torch.equal(a, c) and torch.equal(b, c) and not c.is_inference()
    y = conv()
    (dw,) = torch.autograd.grad(y, w, torch.ones_like(y))
    assert torch.equal(y.detach(), c) and torch.isfinite(dw).all()
    with torch.no_grad():
        w.mul_(2.0)  # an in-place update, as an optimiser's
    with torch.inference_mode():
        d = conv()
    w = w.detach().clone()
    with torch.no_grad():
        assert torch.equal(d, conv()) and not torch.equal(d, c)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_layers_and_weights_made_in_inference_mode(cuda_device, dtype):
    import fvdb
    import fvdb.nn as fvnn

    grid = _grid(fvdb, cuda_device)
    g = torch.Generator().manual_seed(3)
    x = torch.randn(grid.total_voxels, 32, generator=g).to(cuda_device, dtype)
    net = fvnn.Sequential(fvnn.SparseConv3d(32, 16, 3), fvnn.BatchNorm(16), fvnn.ReLU(),
                          fvnn.SparseConv3d(16, 32, 2, stride=2)).to(cuda_device, dtype).eval()
    with torch.inference_mode():
        a = net(fvnn.VDBTensor(grid, x)).data.jdata
        w = net[0].weight * 1.0  # an inference tensor
        pack, _ = grid.sparse_conv_kernel_map(3, 1)
        b = pack.sparse_conv_3d(x, w).jdata
        w.mul_(2.0)  # nothing derived from it may be found again
        b2 = pack.sparse_conv_3d(x, w).jdata
    with torch.no_grad():
        assert torch.equal(a, net(fvnn.VDBTensor(grid, x)).data.jdata)
        assert torch.equal(b, pack.sparse_conv_3d(x, net[0].weight).jdata)
        assert torch.equal(b2, pack.sparse_conv_3d(x, net[0].weight * 2.0).jdata)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_halo_convolution(cuda_device, dtype):
    import fvdb

    grid = _grid(fvdb, cuda_device)
    g = torch.Generator().manual_seed(1)
    w = (torch.randn(32, 64, 3, 3, 3, generator=g) * 0.05).to(cuda_device, dtype).requires_grad_(True)
    x = torch.randn(grid.total_voxels, 64, generator=g).to(cuda_device, dtype)
    with torch.inference_mode():
        a = grid.sparse_conv_halo(grid.jagged_like(x), w).jdata
    with torch.no_grad():
        b = grid.sparse_conv_halo(grid.jagged_like(x), w).jdata
    y = grid.sparse_conv_halo(grid.jagged_like(x), w).jdata
    (dw,) = torch.autograd.grad(y, w, torch.ones_like(y))
    assert torch.equal(a, b) and torch.equal(y.detach(), b) and torch.isfinite(dw).all()


@pytest.mark.parametrize("create_graph", [False, True])
def test_group_norm_trains_on_a_grid_built_in_inference_mode(cuda_device, create_graph):
    import fvdb
    import fvdb.nn as fvnn

    with torch.inference_mode():
        grid = _grid(fvdb, cuda_device)
        assert grid.joffsets.is_inference()
    plain = _grid(fvdb, cuda_device)
    net = fvnn.GroupNorm(4, 16).to(cuda_device)
    g = torch.Generator().manual_seed(4)
    x = torch.randn(grid.total_voxels, 16, generator=g).to(cuda_device).requires_grad_(True)
    dy = torch.randn(grid.total_voxels, 16, generator=g).to(cuda_device)
    got, want = (torch.autograd.grad(net(fvnn.VDBTensor(v, x)).data.jdata, [x, net.weight, net.bias], dy,
                                     create_graph=create_graph) for v in (grid, plain))
    for a, b in zip(got, want):  # the composed operations' sums differ from run to run by FP32 rounding
        assert float((a - b).norm() / b.norm()) <= 1e-4
