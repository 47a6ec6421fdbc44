"""Pooling over a window map equals pooling by lookups, bit for bit: through the C ABI over windows, strides,
types, row widths and grids, and through the package on both sides of the rule that chooses (number of
window positions, voxels per leaf, memory)."""

import ctypes

import numpy as np
import pytest
import torch

from tests.helpers import dense_ijk, random_sparse_ijk

pytestmark = pytest.mark.gpu

MAX, AVG, SUM = 0, 1, 2
DTYPES = {torch.float32: 0, torch.float64: 1, torch.bfloat16: 2, torch.float16: 3}


class Grid(ctypes.Structure):
    _fields_ = [
        ("num_grids", ctypes.c_int32), ("reserved", ctypes.c_int32), ("num_voxels", ctypes.c_int64),
        ("num_leaves", ctypes.c_int64), ("hash_capacity", ctypes.c_int64), ("voxel_offsets", ctypes.c_void_p),
        ("ijk", ctypes.c_void_p), ("leaves", ctypes.c_void_p), ("hash_slots", ctypes.c_void_p),
    ]


def _view(g):
    i = g._impl
    return Grid(i.grid_count, 0, i.total_voxels, i.total_leaf_nodes, i.hash.numel(), i.joffsets.data_ptr(),
                i.ijk.data_ptr(), i.leaves.data_ptr(), i.hash.data_ptr())


def P(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("c", [1, 3, 8, 40])
@pytest.mark.parametrize("window,stride", [((2, 2, 2), (2, 2, 2)), ((3, 3, 3), (2, 2, 2)), ((1, 2, 3), (2, 2, 4)),
                                           ((4, 4, 2), (4, 4, 2))])
def test_map_equals_lookups(cuda_device, dtype, c, window, stride):
    import fvdb
    from fvdb import _lib

    lib = _lib.cdll()
    parts = [random_sparse_ijk(1500, 18, 5, lo=-7), np.zeros((0, 3), np.int32), dense_ijk((9, 6, 11), (3, -4, 0)),
             random_sparse_ijk(40, 600, 6, lo=-300)]
    fine = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor([torch.from_numpy(p).to(cuda_device) for p in parts]))
    coarse = fine.coarsened_grid(list(stride))
    n, W = coarse.total_voxels, int(np.prod(window))
    g = torch.Generator().manual_seed(c)
    x = torch.randn(fine.total_voxels, c, generator=g).to(cuda_device, dtype)
    f, cv = _view(fine), _view(coarse)
    w, st = (ctypes.c_int32 * 3)(*window), (ctypes.c_int32 * 3)(*stride)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    m = torch.full((n, W), -9, dtype=torch.int32, device=cuda_device)
    assert lib.fvgb_window_map(ctypes.byref(f), ctypes.byref(cv), w, st, P(m), s) == 0
    i64 = ctypes.c_int64
    for mode in (MAX, AVG, SUM):
        a, b = (torch.full((n, c), 7.0, device=cuda_device, dtype=dtype) for _ in range(2))
        assert lib.fvgb_pool_forward_map(mode, DTYPES[dtype], P(m), i64(n), W, P(x), i64(c), c, P(a), i64(c), s) == 0
        if mode == SUM:
            if window != stride:
                continue
            assert lib.fvgb_upsample_backward(DTYPES[dtype], ctypes.byref(cv), ctypes.byref(f), w, P(x), i64(c), c, P(b),
                                              i64(c), s) == 0
        else:
            assert lib.fvgb_pool_forward(mode, DTYPES[dtype], ctypes.byref(f), ctypes.byref(cv), w, st, P(x), i64(c), c,
                                         P(b), i64(c), s) == 0
        torch.cuda.synchronize()
        assert torch.equal(a, b)
    if all(q >= p for p, q in zip(window, stride)):
        dy = torch.randn(n, c, generator=g).to(cuda_device, dtype)
        dx = torch.zeros_like(x)
        assert lib.fvgb_maxpool_backward_map(DTYPES[dtype], P(m), i64(n), W, P(x), i64(c), c, P(dy), i64(c), P(dx), s) == 0
        acc = torch.zeros(x.shape, device=cuda_device, dtype=torch.float64 if dtype == torch.float64 else torch.float32)
        assert lib.fvgb_maxpool_backward(DTYPES[dtype], ctypes.byref(f), ctypes.byref(cv), w, st, P(x), i64(c), c, P(dy),
                                         i64(c), P(acc), s) == 0
        torch.cuda.synchronize()
        assert torch.equal(dx, acc.to(dtype))


def _reference(grid, coarse, f, x, dy):
    """Max over disjoint f^3 windows, its gradient (to the first maximum in window order) and the sum of a
    coarse voxel's children, with torch operations."""
    parent = coarse.ijk_to_index(grid.jagged_like(torch.div(grid.ijk.jdata, f, rounding_mode="floor")), cumulative=True).jdata
    at = grid.ijk.jdata.long() % f
    pos = (at[:, 0] * f + at[:, 1]) * f + at[:, 2]
    full = x.new_full((coarse.total_voxels, f**3, x.shape[1]), float("-inf"))
    full[parent, pos] = x
    y, arg = full.amax(1), (full == full.amax(1, keepdim=True)).to(torch.uint8).argmax(1)
    dx = torch.where(arg[parent] == pos[:, None], dy[parent], torch.zeros_like(x))
    total = torch.zeros(coarse.total_voxels, x.shape[1], dtype=torch.float64, device=x.device).index_add_(0, parent, x.double())
    return y, dx, total


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("kind,f", [("surface", 2), ("scattered", 2), ("dense", 2), ("dense", 3)])
def test_both_sides_of_the_rule(cuda_device, dtype, kind, f):
    import fvdb

    g = torch.Generator().manual_seed(2)
    if kind == "surface":  # 2.3M positions over the coarse grid, about 50 voxels per leaf
        p = torch.randn(4_500_000, 3, generator=g)
        ijk = (p / p.norm(dim=1, keepdim=True) * 270).round().int()
    elif kind == "scattered":  # as many positions, one voxel per leaf
        ijk = torch.randint(-8000, 8000, (300_000, 3), generator=g, dtype=torch.int32)
    else:
        ijk = torch.from_numpy(dense_ijk((104, 104, 104), (-3, 5, -50)))
    grid = fvdb.GridBatch.from_ijk(ijk.to(cuda_device))
    coarse = grid.coarsened_grid(f)
    x = torch.randint(-8, 9, (grid.total_voxels, 8), generator=g).to(cuda_device, dtype)
    dy = torch.randint(-8, 9, (coarse.total_voxels, 8), generator=g).to(cuda_device, dtype)
    y_ref, dx_ref, total = _reference(grid, coarse, f, x, dy)
    xr = x.clone().requires_grad_(True)
    y = grid.max_pool(f, grid.jagged_like(xr), coarse_grid=coarse)[0].jdata
    y.backward(dy)
    assert torch.equal(y.detach(), y_ref) and torch.equal(xr.grad, dx_ref)
    z = dy.clone().requires_grad_(True)
    up = coarse.subdivide(f, coarse.jagged_like(z), fine_grid=grid)[0].jdata
    up.backward(x)
    assert torch.equal(z.grad.double(), total)  # whole numbers below 2^8


def test_without_memory_for_the_map(cuda_device):
    import fvdb

    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(dense_ijk((128, 128, 128))).to(cuda_device))
    coarse = grid.coarsened_grid(1)  # 2.1M windows of 27 positions: 226 MB of map
    x = grid.jagged_like(torch.randn(grid.total_voxels, 4, device=cuda_device))
    want = grid.max_pool(3, x, stride=1, coarse_grid=coarse)[0].jdata
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (100 << 20)) / total)
        got = grid.max_pool(3, x, stride=1, coarse_grid=coarse)[0].jdata
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)
