"""sparse_conv_halo over a kernel map and on the leaf kernels, each asked for by itself, against the FP64
oracle: every type, channels that are and are not multiples of 8, leaf borders, scattered voxels and
several grids; and calls near the sizes where the route changes, without memory for the map, and among
convolutions whose packed weights are kept.

Tolerances (relative L2): FP32 accumulation (1e-5; 1e-12 in FP64) and one rounding of 16-bit results."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.helpers import dense_ijk, random_sparse_ijk

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def f64(t):
    return t.detach().double().cpu().numpy()


def _lim(dtype):
    return 1e-12 if dtype == torch.float64 else 1e-5 + (torch.finfo(dtype).eps / 2 if dtype.itemsize == 2 else 0.0)


def _oracle(grid, x, w, dy):
    """y, dx, dW [27, I, O] in FP64 for weights [27, I, O]"""
    v, off = grid.ijk.jdata.cpu().numpy(), grid.joffsets.cpu().numpy()
    kmap = orc.kernel_map(v, off, v, off, 3, 1)
    w5 = f64(w).reshape(3, 3, 3, w.shape[1], w.shape[2]).transpose(4, 3, 2, 1, 0)
    y = orc.conv_forward_f64(f64(x), w5, kmap)
    dx, dw = orc.conv_backward_f64(f64(x), w5, kmap, f64(dy))
    return y, dx, dw.transpose(4, 3, 2, 1, 0).reshape(27, w.shape[1], w.shape[2])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cin,cout", [(8, 16), (24, 40), (3, 5), (64, 32), (33, 8)])
def test_each_route(cuda_device, dtype, cin, cout):
    import fvdb
    from fvdb import _lib

    C = _lib.load()
    parts = [dense_ijk((17, 9, 11), (-5, 3, -2)), random_sparse_ijk(700, 20, 3, lo=-9), random_sparse_ijk(60, 500, 4)]
    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor([torch.from_numpy(p).to(cuda_device) for p in parts]))
    g = torch.Generator().manual_seed(cin)
    x = torch.randn(grid.total_voxels, cin, generator=g).to(cuda_device, dtype)
    w = (torch.randn(27, cin, cout, generator=g) / (27 * cin) ** 0.5).to(cuda_device, dtype)
    dy = torch.randn(grid.total_voxels, cout, generator=g).to(cuda_device, dtype)
    y_ref, dx_ref, dw_ref = _oracle(grid, x, w, dy)
    for route in (C.HALO_LEAF, C.HALO_MAP):
        y = C.halo_conv(grid._impl, x, w, False, route)
        dx = C.halo_conv(grid._impl, dy, w, True, route)
        dw = C.halo_wgrad(grid._impl, x, dy, route)
        assert y.dtype == dx.dtype == dw.dtype == dtype
        assert rel(f64(y), y_ref) <= _lim(dtype)
        assert rel(f64(dx), dx_ref) <= _lim(dtype)
        assert rel(f64(dw), dw_ref) <= _lim(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [2047, 2048, 4095, 4096, 16383, 16384])
@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 24), (24, 24)])
def test_both_sides_of_the_rule(cuda_device, dtype, n, cin, cout):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(dense_ijk((32, 32, 16))[:n]).to(cuda_device))
    g = torch.Generator().manual_seed(n)
    x = torch.randn(n, cin, generator=g).to(cuda_device, dtype).requires_grad_(True)
    w = (torch.randn(cout, cin, 3, 3, 3, generator=g) / (27 * cin) ** 0.5).to(cuda_device, dtype).requires_grad_(True)
    dy = torch.randn(n, cout, generator=g).to(cuda_device, dtype)
    y = grid.sparse_conv_halo(grid.jagged_like(x), w).jdata
    dx, dw = torch.autograd.grad(y, [x, w], dy)
    wk = w.detach().permute(4, 3, 2, 1, 0).reshape(27, cin, cout)
    y_ref, dx_ref, dw_ref = _oracle(grid, x, wk, dy)
    for a, b in ((y, y_ref), (dx, dx_ref), (dw.permute(4, 3, 2, 1, 0).reshape(27, cin, cout), dw_ref)):
        assert rel(f64(a), b) <= _lim(dtype)


def test_without_memory_for_the_map(cuda_device):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(dense_ijk((128, 128, 128))).to(cuda_device))
    n = grid.total_voxels  # 226 MB of map
    x = torch.randn(n, 16, device=cuda_device).bfloat16()
    w = (torch.randn(16, 16, 3, 3, 3, device=cuda_device) * 0.05).bfloat16()
    want = grid.sparse_conv_halo(grid.jagged_like(x), w).jdata
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    got = []
    try:
        for extra in (80, 310):  # room for the output alone; for the map too, but not for what goes with it
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (extra << 20)) / total)
            got.append(grid.sparse_conv_halo(grid.jagged_like(x), w).jdata.cpu())
            torch.cuda.empty_cache()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for y in got:
        assert rel(f64(y), f64(want)) <= 2 * _lim(torch.bfloat16)


def test_packed_weights_of_other_layers_stay(cuda_device):
    import fvdb
    from fvdb import _lib

    count = _lib.cdll().fvgb_launch_count
    count.restype = ctypes.c_uint64
    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(3000, 24, 1)).to(cuda_device))
    pack, _ = grid.sparse_conv_kernel_map(3, 1)
    x = torch.randn(grid.total_voxels, 32, device=cuda_device).bfloat16()
    w = (torch.randn(64, 32, 3, 3, 3, device=cuda_device) * 0.05).bfloat16()

    def launches():
        a = count()
        pack.sparse_conv_3d(x, w)
        return count() - a

    for _ in range(3):
        warm = launches()
    for _ in range(70):
        grid.sparse_conv_halo(grid.jagged_like(x), w)
    assert launches() == warm
