"""Gradients of several output vectors at once (autograd.grad with is_grads_batched, a vectorised
jacobian, torch.func.vmap over a backward pass) equal a loop over the vectors.  The batched gradient
that a backward function sees has no memory a kernel could read."""

import pytest
import torch

from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu

DTYPE, TOL = torch.float64, dict(rtol=1e-10, atol=1e-10)  # FP64 arithmetic in another order


def _compare(y, ins, vs):
    want = [torch.stack(t) for t in zip(*[torch.autograd.grad(y, ins, v, retain_graph=True) for v in vs])]
    batched = torch.autograd.grad(y, ins, vs, retain_graph=True, is_grads_batched=True)
    mapped = torch.func.vmap(lambda v: torch.autograd.grad(y, ins, v, retain_graph=True))(vs)
    for a, b, c in zip(want, batched, mapped):
        torch.testing.assert_close(b, a, **TOL)
        torch.testing.assert_close(c, a, **TOL)


@pytest.mark.parametrize("frozen", [False, True])
def test_group_norm(cuda_device, frozen):
    import fvdb
    import fvdb.nn as fvnn

    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor([torch.from_numpy(random_sparse_ijk(n, 16, n)).to(cuda_device)
                                                      for n in (70, 40)]))
    net = fvnn.GroupNorm(2, 8).to(cuda_device, DTYPE).requires_grad_(not frozen)
    leaf = torch.randn(grid.total_voxels, 8, device=cuda_device, dtype=DTYPE, requires_grad=True)
    y = net(fvnn.VDBTensor(grid, leaf * 1.5 + 0.2)).data.jdata
    _compare(y, [leaf] if frozen else [leaf, net.weight, net.bias], torch.randn(3, *y.shape, device=cuda_device, dtype=DTYPE))
    rows = torch.autograd.functional.jacobian(lambda t: net(fvnn.VDBTensor(grid, t)).data.jdata[:2], leaf.detach(),
                                              vectorize=True)
    loop = torch.autograd.functional.jacobian(lambda t: net(fvnn.VDBTensor(grid, t)).data.jdata[:2], leaf.detach())
    torch.testing.assert_close(rows, loop, **TOL)


@pytest.mark.parametrize("relu", [False, True])
def test_convolution_whose_bias_alone_needs_a_gradient(cuda_device, relu):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(200, 12, 1)).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    x = torch.randn(grid.total_voxels, 4, device=cuda_device, dtype=DTYPE)
    w = torch.randn(6, 4, 3, 3, 3, device=cuda_device, dtype=DTYPE)
    b = torch.randn(6, device=cuda_device, dtype=DTYPE, requires_grad=True)
    y = pack._conv_with_bias(x, w, b, False, None, relu).jdata
    _compare(y, [b], torch.randn(3, *y.shape, device=cuda_device, dtype=DTYPE))
