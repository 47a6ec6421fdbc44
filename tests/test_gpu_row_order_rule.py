"""When a contraction takes a map's row order: at the first use of a large map that will be used again, at
the second use of any, and never where memory does not allow it; with the same outputs bit for bit."""

import pytest
import torch

from tests.helpers import dense_ijk, random_sparse_ijk

pytestmark = pytest.mark.gpu


def _case(dev, n, cin, cout, ks=3, st=1, dense=False, transposed=False):
    import fvdb

    ijk = dense_ijk((48, 48, (n + 2303) // 2304))[:n] if dense else random_sparse_ijk(n, 96, 5)
    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(ijk).to(dev))
    pack, tgt = grid.sparse_conv_kernel_map(ks, st)
    g = torch.Generator().manual_seed(n)
    rows = tgt.total_voxels if transposed else grid.total_voxels
    x = torch.randn(rows, cin, generator=g).to(dev, torch.bfloat16)
    shape = (cin, cout) if transposed else (cout, cin)
    w = (torch.randn(*shape, ks, ks, ks, generator=g) * 0.05).to(dev, torch.bfloat16)
    return grid, pack, x, w


def _step(pack, x, w):
    xr, wr = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    y = pack.sparse_conv_3d(xr, wr).jdata
    return [y.detach(), *torch.autograd.grad(y, [xr, wr], torch.ones_like(y))]


@pytest.mark.parametrize("n", [(1 << 16) - 1, 1 << 16])
def test_training_step(cuda_device, n):
    grid, pack, x, w = _case(cuda_device, n, 32, 64)
    first = _step(pack, x, w)
    assert pack._impl.has_row_order() == (n >= 1 << 16)
    second = _step(pack, x, w)  # the map's second forward contraction
    assert pack._impl.has_row_order()
    assert torch.equal(first[0], second[0]) and torch.equal(first[1], second[1])
    assert torch.equal(first[2], second[2])


def test_training_step_over_scattered_voxels(cuda_device):
    import fvdb

    g = torch.Generator().manual_seed(1)
    ijk = torch.randint(-4000, 4000, (70000, 3), generator=g, dtype=torch.int32)
    grid = fvdb.GridBatch.from_ijk(ijk.to(cuda_device))
    assert 1 << 16 <= grid.total_voxels < 2 * grid._impl.total_leaf_nodes
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    x = torch.randn(grid.total_voxels, 32, generator=g).to(cuda_device, torch.bfloat16)
    w = (torch.randn(64, 32, 3, 3, 3, generator=g) * 0.05).to(cuda_device, torch.bfloat16)
    first = _step(pack, x, w)
    assert not pack._impl.has_row_order()
    second = _step(pack, x, w)
    assert pack._impl.has_row_order()
    assert torch.equal(first[0], second[0]) and torch.equal(first[1], second[1])


@pytest.mark.parametrize("n,cin,cout,dense,at_once", [
    ((1 << 18) - 1, 128, 128, False, False), (1 << 18, 128, 128, False, True), (1 << 18, 64, 256, False, False),
    (1 << 18, 128, 128, True, False), (1 << 18, 128, 64, False, False)])
def test_wide_layers(cuda_device, n, cin, cout, dense, at_once):
    grid, pack, x, w = _case(cuda_device, n, cin, cout, dense=dense)
    a = pack.sparse_conv_3d(x, w).jdata
    assert pack._impl.has_row_order() == at_once
    b = pack.sparse_conv_3d(x, w).jdata
    assert pack._impl.has_row_order() and torch.equal(a, b)


@pytest.mark.parametrize("n,cin,at_once", [(65535, 256, False), (65536, 256, True), (65536, 128, False), (200000, 64, False)])
def test_transposed_maps_of_one_entry(cuda_device, n, cin, at_once):
    grid, pack, x, w = _case(cuda_device, n, cin, 32, ks=2, st=2, transposed=True)
    a = pack.sparse_transpose_conv_3d(x, w).jdata
    assert pack._impl.has_row_order(True) == at_once
    b = pack.sparse_transpose_conv_3d(x, w).jdata
    assert pack._impl.has_row_order(True) and torch.equal(a, b)


@pytest.mark.parametrize("n,cin,at_once", [((1 << 19) - 1, 64, False), (1 << 19, 64, True), (1 << 19, 32, False)])
def test_transposed_maps_of_one_entry_in_training(cuda_device, n, cin, at_once):
    grid, pack, x, w = _case(cuda_device, n, cin, 32, ks=2, st=2, transposed=True)
    grads = []
    for use in range(2):
        xr, wr = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
        y = pack.sparse_transpose_conv_3d(xr, wr).jdata
        assert pack._impl.has_row_order(True) == (at_once or use == 1)
        y.backward(torch.ones_like(y))
        grads.append((y.detach(), xr.grad, wr.grad))
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_without_memory_for_the_order(cuda_device):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(dense_ijk((128, 128, 96))).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    x = torch.randn(grid.total_voxels, 16, device=cuda_device).bfloat16()
    w = (torch.randn(16, 16, 3, 3, 3, device=cuda_device) * 0.05).bfloat16()
    want = pack.sparse_conv_3d(x, w).jdata
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    try:  # the output takes 50 MB, the order 170
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (80 << 20)) / total)
        got = pack.sparse_conv_3d(x, w).jdata
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want) and not pack._impl.has_row_order()
    assert torch.equal(pack.sparse_conv_3d(x, w).jdata, want) and pack._impl.has_row_order()


@pytest.mark.parametrize("ks,st,transposed", [(3, 1, False), (3, 1, True), (2, 2, False), (2, 2, True)])
@pytest.mark.parametrize("n", [6000, 1 << 16])
@pytest.mark.parametrize("features_too", [True, False])
def test_weight_gradient_is_the_same_whether_the_order_is_built(cuda_device, ks, st, transposed, n, features_too):
    grid, pack, x, w = _case(cuda_device, n, 32, 64, ks, st, transposed=transposed)
    conv = pack.sparse_transpose_conv_3d if transposed else pack.sparse_conv_3d
    g = torch.Generator().manual_seed(3)
    grads = []
    for use in range(3):
        wr = w.clone().requires_grad_(True)
        y = conv(x.clone().requires_grad_(features_too), wr).jdata
        if use == 0:
            dy = torch.randn(y.shape, generator=g).to(cuda_device, torch.bfloat16)
        y.backward(dy)
        grads.append(wr.grad)
    impl = pack._impl
    assert impl.has_row_order(False) or impl.has_row_order(True)
    assert torch.equal(grads[0], grads[1]) and torch.equal(grads[0], grads[2])
