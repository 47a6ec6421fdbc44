"""GPU parity of pooling and nearest upsampling (fvdb.nn.MaxPool / AvgPool / UpsamplingNearest)
against the oracle: grids (coarsened / subdivided) bit-exact, FP32 and FP64 values and gradients
bit-exact where the reference is deterministic (non-overlapping windows), BF16 within 1e-2 of
the oracle on the same rounded inputs, overlapping windows within 1e-6 (FP32; summation order)."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fvdb(cuda_device):
    import fvdb as m

    return m


def _grid(fvdb, dev, seeds=(1, 2), n=3000, extent=24):
    parts = [random_sparse_ijk(n, extent, s, lo=-10 * s) for s in seeds]
    ijk = np.concatenate(parts)
    off = np.cumsum([0] + [p.shape[0] for p in parts])
    jt = fvdb.JaggedTensor.from_data_and_offsets(torch.from_numpy(ijk).to(dev), torch.from_numpy(off).to(dev))
    g = fvdb.GridBatch.from_ijk(jt)
    return g, g.ijk.jdata.cpu().numpy(), g.joffsets.cpu().numpy()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("pool,stride", [(2, 0), ((2, 3, 1), 0), (3, 4), (2, (2, 3, 2))])
def test_pool_bit_exact(fvdb, cuda_device, dtype, mode, pool, stride):
    g, ijk, off = _grid(fvdb, cuda_device)
    x = torch.randn(g.total_voxels, 5, dtype=dtype, generator=torch.Generator().manual_seed(3))
    xd = x.to(cuda_device).requires_grad_(True)
    fn = g.max_pool if mode == "max" else g.avg_pool
    y, cg = fn(pool, fvdb.JaggedTensor.from_data_and_offsets(xd, g.joffsets), stride=stride)
    st = stride if stride else pool
    c_o, coff_o = orc.coarsened_grid(ijk, off, st)
    c = cg.ijk.jdata.cpu().numpy()
    assert np.array_equal(c, c_o) and np.array_equal(cg.joffsets.cpu().numpy(), coff_o)
    ref = orc.pool_forward(ijk, off, c, coff_o, x.numpy(), pool, stride, mode)
    assert np.array_equal(y.jdata.detach().cpu().numpy(), ref)
    dy = torch.randn(y.jdata.shape, dtype=dtype, generator=torch.Generator().manual_seed(4))
    y.jdata.backward(dy.to(cuda_device))
    ref_dx = orc.pool_backward(ijk, off, c, coff_o, x.numpy(), dy.numpy(), pool, stride, mode)
    assert np.array_equal(xd.grad.cpu().numpy(), ref_dx)


def test_overlapping_windows_and_user_coarse_grid(fvdb, cuda_device):
    g, ijk, off = _grid(fvdb, cuda_device)
    cg = g.coarsened_grid(2)  # stride 2 with a 3-wide window: windows overlap
    x = torch.randn(g.total_voxels, 4, generator=torch.Generator().manual_seed(5))
    xd = x.to(cuda_device).requires_grad_(True)
    y, out_grid = g.avg_pool(3, fvdb.JaggedTensor.from_data_and_offsets(xd, g.joffsets), stride=2, coarse_grid=cg)
    assert out_grid.is_same(cg)
    c, coff = cg.ijk.jdata.cpu().numpy(), cg.joffsets.cpu().numpy()
    ref = orc.pool_forward(ijk, off, c, coff, x.numpy(), 3, 2, "avg")
    assert np.array_equal(y.jdata.detach().cpu().numpy(), ref)
    dy = torch.randn(y.jdata.shape, generator=torch.Generator().manual_seed(6))
    y.jdata.backward(dy.to(cuda_device))
    ref_dx = orc.pool_backward(ijk, off, c, coff, x.numpy(), dy.numpy(), 3, 2, "avg")
    np.testing.assert_allclose(xd.grad.cpu().numpy(), ref_dx, rtol=1e-6, atol=1e-6)


def test_bf16_pool_and_modules(fvdb, cuda_device):
    g, ijk, off = _grid(fvdb, cuda_device)
    x = torch.randn(g.total_voxels, 8, generator=torch.Generator().manual_seed(7)).bfloat16()
    vt = fvdb.nn.VDBTensor(g, g.jagged_like(x.to(cuda_device)))
    out = fvdb.nn.MaxPool(2)(vt)
    c, coff = out.grid.ijk.jdata.cpu().numpy(), out.grid.joffsets.cpu().numpy()
    ref = orc.pool_forward(ijk, off, c, coff, x.float().numpy(), 2, 0, "max")
    assert np.array_equal(out.data.jdata.float().cpu().numpy(), ref)  # max of bf16 values is exact
    avg = fvdb.nn.AvgPool(2)(vt)
    ref_a = orc.pool_forward(ijk, off, c, coff, x.float().numpy(), 2, 0, "avg")
    np.testing.assert_allclose(avg.data.jdata.float().cpu().numpy(), ref_a, rtol=1e-2, atol=1e-2)
    # coarse transform as the reference: size 2w, origin o + w/2
    assert torch.allclose(out.grid.voxel_sizes[0], g.voxel_sizes[0] * 2)
    assert torch.allclose(out.grid.origins[0], g.origins[0] + 0.5 * g.voxel_sizes[0])


def test_maxpool_module_zeroes_empty_windows(fvdb, cuda_device):
    src = fvdb.GridBatch.from_ijk(torch.tensor([[0, 0, 0], [1, 1, 1]], dtype=torch.int32, device=cuda_device))
    coarse = fvdb.GridBatch.from_ijk(torch.tensor([[0, 0, 0], [5, 5, 5]], dtype=torch.int32, device=cuda_device))
    vt = fvdb.nn.VDBTensor(src, src.jagged_like(torch.tensor([[1.0], [-3.0]], device=cuda_device)))
    raw, _ = src.max_pool(2, vt.data, coarse_grid=coarse)
    assert torch.isinf(raw.jdata[1]).all() and raw.jdata[1, 0] < 0
    out = fvdb.nn.MaxPool(2)(vt, coarse)
    assert out.data.jdata[:, 0].tolist() == [1.0, 0.0]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("factor,masked", [(2, False), ((1, 2, 3), True)])
def test_upsample_bit_exact(fvdb, cuda_device, dtype, factor, masked):
    g, ijk, off = _grid(fvdb, cuda_device, n=800, extent=16)
    mask = None
    if masked:
        mask = torch.rand(g.total_voxels, generator=torch.Generator().manual_seed(8)) < 0.6
    x = torch.randn(g.total_voxels, 3, dtype=dtype, generator=torch.Generator().manual_seed(9))
    xd = x.to(cuda_device).requires_grad_(True)
    y, fg = g.subdivide(factor, fvdb.JaggedTensor.from_data_and_offsets(xd, g.joffsets),
                        mask=None if mask is None else mask.to(cuda_device))
    f_o, foff_o = orc.subdivided_grid(ijk, off, factor, None if mask is None else mask.numpy())
    f = fg.ijk.jdata.cpu().numpy()
    assert np.array_equal(f, f_o) and np.array_equal(fg.joffsets.cpu().numpy(), foff_o)
    assert np.array_equal(y.jdata.detach().cpu().numpy(), orc.upsample_forward(ijk, off, f, foff_o, x.numpy(), factor))
    dy = torch.randn(y.jdata.shape, dtype=dtype, generator=torch.Generator().manual_seed(10))
    y.jdata.backward(dy.to(cuda_device))
    assert np.array_equal(xd.grad.cpu().numpy(), orc.upsample_backward(ijk, off, f, foff_o, dy.numpy(), factor))
    # fine transform as the reference: size w/f, origin o - (f-1) w / (2f)
    fv = torch.tensor(orc._vec3(factor), dtype=torch.float64)
    vs, org = g.voxel_sizes[0].cpu().double(), g.origins[0].cpu().double()
    assert torch.allclose(fg.voxel_sizes[0].cpu().double(), vs / fv)
    assert torch.allclose(fg.origins[0].cpu().double(), org - (fv - 1) * vs / fv * 0.5)


def test_upsample_module_onto_user_grid(fvdb, cuda_device):
    coarse = fvdb.GridBatch.from_ijk(torch.tensor([[0, 0, 0]], dtype=torch.int32, device=cuda_device))
    fine = fvdb.GridBatch.from_ijk(torch.tensor([[1, 1, 1], [4, 4, 4]], dtype=torch.int32, device=cuda_device))
    vt = fvdb.nn.VDBTensor(coarse, coarse.jagged_like(torch.tensor([[2.5, -1.0]], device=cuda_device)))
    out = fvdb.nn.UpsamplingNearest(2)(vt, ref_fine_data=fine)
    assert out.grid.is_same(fine)
    # (1,1,1) has parent (0,0,0); (4,4,4) has none and reads zero
    assert out.data.jdata.cpu().tolist() == [[2.5, -1.0], [0.0, 0.0]]


@pytest.mark.parametrize("c,dtype", [(1, torch.float32), (8, torch.float32), (24, torch.float64), (264, torch.float32),
                                     (8, torch.bfloat16), (40, torch.float16), (20, torch.bfloat16), (272, torch.bfloat16)])
@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("pool,stride", [(2, 0), (3, 4), (8, 0)])
def test_pool_and_upsampling_row_widths(fvdb, cuda_device, c, dtype, mode, pool, stride):
    """Rows of one vector, of a lane group's vectors, of more than a warp's and of single elements;
    windows of 8, 27 and 512; whole numbers, which every type adds exactly: equal to the oracle
    (upsampling where the grids' factor is the pooling factor)."""
    g, ijk, off = _grid(fvdb, cuda_device, n=700)
    gen = torch.Generator().manual_seed(c)
    x = torch.randint(-8, 9, (g.total_voxels, c), generator=gen).to(dtype)
    if mode == "avg" and pool == 3:
        x.zero_()  # 1/27 is not exact in 16 bits; zeros check the windows
    xd = x.to(cuda_device).requires_grad_(True)
    fn = g.max_pool if mode == "max" else g.avg_pool
    y, cg = fn(pool, g.jagged_like(xd), stride=stride)
    st = stride if stride else pool
    cijk, coff = cg.ijk.jdata.cpu().numpy(), cg.joffsets.cpu().numpy()
    ref = orc.pool_forward(ijk, off, cijk, coff, x.double().numpy(), pool, stride, mode)
    assert np.array_equal(y.jdata.detach().double().cpu().numpy(), ref)
    dy = torch.randint(-8, 9, y.jdata.shape, generator=gen).to(dtype)
    y.jdata.backward(dy.to(cuda_device))
    if not (mode == "avg" and pool == 3):
        ref_dx = orc.pool_backward(ijk, off, cijk, coff, x.double().numpy(), dy.double().numpy(), pool, stride, mode)
        assert np.array_equal(xd.grad.double().cpu().numpy(), ref_dx)
    if stride:
        return
    z = dy.to(cuda_device).requires_grad_(True)
    up, _ = cg.subdivide(pool, cg.jagged_like(z), fine_grid=g)
    parent = torch.from_numpy(np.concatenate(
        [np.full(off[b + 1] - off[b], b) for b in range(len(off) - 1)])).to(cuda_device)
    key = torch.cat([parent[:, None], torch.div(g.ijk.jdata, pool, rounding_mode="floor")], 1)
    ckey = torch.cat([cg.jidx.long()[:, None], cg.ijk.jdata], 1)
    _, inv = torch.unique(torch.cat([ckey, key]), dim=0, return_inverse=True)
    row = torch.empty(int(inv.max()) + 1, dtype=torch.long, device=cuda_device)
    row[inv[:ckey.shape[0]]] = torch.arange(ckey.shape[0], device=cuda_device)
    rows = row[inv[ckey.shape[0]:]]
    assert torch.equal(up.jdata, z.detach()[rows])
    ones = torch.ones_like(up.jdata)
    up.jdata.backward(ones)
    assert torch.equal(z.grad.double(), torch.bincount(rows, minlength=z.shape[0]).double()[:, None].expand_as(z))
