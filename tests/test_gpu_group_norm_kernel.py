"""The GroupNorm kernels over their dispatch: every vector width (channels per group a multiple of
8, 4, 2 or odd), channel counts beyond one CTA's columns, chunks that hold several grids, single
voxels and empty grids, all types; against torch.nn.GroupNorm in FP64 grid by grid.

Tolerances (relative L2): 16-bit outputs round once to their type (its unit roundoff, eps / 2, per
value) on top of FP32 arithmetic (1e-5, 1e-12 in FP64); gradients are allowed ten times that term,
as they subtract sums of the same size."""

import pytest
import torch

from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu

ROUND = {torch.float32: 0.0, torch.float64: 0.0, torch.bfloat16: torch.finfo(torch.bfloat16).eps / 2,
         torch.float16: torch.finfo(torch.float16).eps / 2}


def rel(a, b):
    a, b = a.detach().double(), b.detach().double()
    return float((a - b).norm() / b.norm().clamp(min=1e-30))


def _case(fvdb, dev, sizes, c, dtype, seed=5):
    parts = [torch.from_numpy(random_sparse_ijk(n, 24, seed + i)).to(dev) if n else
             torch.zeros((0, 3), dtype=torch.int32, device=dev) for i, n in enumerate(sizes)]
    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor(parts))
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(grid.total_voxels, c, generator=g) * 2 + 0.7).to(dev, dtype)
    dy = torch.randn(grid.total_voxels, c, generator=g).to(dev, dtype)
    return grid, x, dy, g


def _reference(grid, x, dy, net):
    x64 = x.detach().double().requires_grad_(True)
    w, b = (net.weight.detach().double().requires_grad_(True), net.bias.detach().double().requires_grad_(True))
    off = grid.joffsets.tolist()
    ys = [torch.nn.functional.group_norm(x64[s:e].t()[None], net.num_groups, w, b, net.eps)[0].t()
          for s, e in zip(off[:-1], off[1:]) if e > s]
    y = torch.cat(ys)
    return (y, *torch.autograd.grad(y, [x64, w, b], dy.double()))


@pytest.mark.parametrize("c,groups,sizes,dtype", [
    (64, 8, [3000, 0, 700, 1, 255], torch.bfloat16),
    (48, 16, [257, 513], torch.float16),
    (96, 8, [2049], torch.bfloat16),
    (16, 4, [5, 1, 1, 600, 0, 2], torch.float32),
    (24, 8, [1200, 40], torch.bfloat16),
    (6, 2, [900, 300], torch.float64),
    (1030, 2, [70, 9], torch.float32),
    (4096, 4, [33], torch.bfloat16),
])
def test_group_norm_kernel(cuda_device, c, groups, sizes, dtype):
    import fvdb
    import fvdb.nn as fvnn

    grid, x, dy, g = _case(fvdb, cuda_device, sizes, c, dtype)
    net = fvnn.GroupNorm(groups, c).to(cuda_device, dtype)
    with torch.no_grad():
        net.weight.copy_(torch.rand(c, generator=g) + 0.5)
        net.bias.copy_(torch.randn(c, generator=g))
    xr = x.requires_grad_(True)
    y = net(fvnn.VDBTensor(grid, xr)).data.jdata
    got = (y, *torch.autograd.grad(y, [xr, net.weight, net.bias], dy))
    again = net(fvnn.VDBTensor(grid, xr)).data.jdata
    assert torch.equal(y, again)
    base = 1e-12 if dtype == torch.float64 else 1e-5
    for i, (a, b) in enumerate(zip(got, _reference(grid, x, dy, net))):
        assert a.dtype == dtype
        assert rel(a, b) <= ROUND[dtype] + base * (1 if i == 0 else 10)


def test_group_norm_strided_rows_and_second_derivative(cuda_device):
    import fvdb
    import fvdb.nn as fvnn

    grid, x, dy, _ = _case(fvdb, cuda_device, [60, 20], 8, torch.float64)
    net = fvnn.GroupNorm(2, 8).to(cuda_device, torch.float64)
    wide = torch.randn(grid.total_voxels, 16, device=cuda_device, dtype=torch.float64)
    assert torch.equal(net(fvnn.VDBTensor(grid, wide[:, ::2])).data.jdata,
                       net(fvnn.VDBTensor(grid, wide[:, ::2].contiguous())).data.jdata)

    def f(t):
        return net(fvnn.VDBTensor(grid, t)).data.jdata

    def composed(t):
        from fvdb._norm import group_norm_composed

        return group_norm_composed(t, grid.jidx.long(), 2, 2, net.eps, net.weight, net.bias)

    def second(fn):
        t = x.detach().requires_grad_(True)
        (gx,) = torch.autograd.grad(fn(t), t, dy, create_graph=True)
        return torch.autograd.grad(gx.square().sum(), [t, net.weight])

    for a, b in zip(second(f), second(composed)):
        assert rel(a, b) <= 1e-10
    _, t = torch.func.jvp(f, (x.detach(),), (dy,))
    (v,) = torch.func.vjp(f, x.detach())[1](dy)
    assert torch.isfinite(t).all() and torch.isfinite(v).all()
