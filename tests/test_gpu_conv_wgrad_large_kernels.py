"""Weight gradients on the tensor cores for kernels of more than 32 offsets, whose map rows are not
staged beside the output gradient: the warps that gather the other operand run ahead of its tiles, and
a tile's buffer may only be reused when the products over it are done.  125 offsets at these channel
counts leave the last block of offsets a single group of them, so the gathers can be three tiles ahead.

Tolerance (relative L2): FP32 accumulation (2e-5) and one rounding of the result (eps / 2)."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.helpers import dense_ijk, random_sparse_ijk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,dtype", [(128, 256, torch.bfloat16), (64, 256, torch.float16), (128, 128, torch.bfloat16),
                                            (8, 8, torch.float16)])
@pytest.mark.parametrize("dense", [True, False])
def test_weight_gradient_of_125_offsets(cuda_device, cin, cout, dtype, dense):
    import fvdb

    ijk = dense_ijk((20, 20, 21)) if dense else random_sparse_ijk(9001, 40, 7)
    grid = fvdb.GridBatch.from_ijk(torch.from_numpy(ijk).to(cuda_device))
    n = grid.total_voxels
    pack, _ = grid.sparse_conv_kernel_map(5, 1)
    g = torch.Generator().manual_seed(cin)
    x = torch.randn(n, cin, generator=g).to(cuda_device, dtype)
    w = torch.zeros(cout, cin, 5, 5, 5, device=cuda_device, dtype=dtype, requires_grad=True)
    dy = torch.randn(n, cout, generator=g).to(cuda_device, dtype)
    v = grid.ijk.jdata.cpu().numpy()
    off = np.array([0, n])
    kmap = torch.from_numpy(orc.kernel_map(v, off, v, off, 5, 1)).to(cuda_device).long()
    want = torch.stack([x[kmap[:, k].clamp(min=0)].double().mul((kmap[:, k] >= 0)[:, None]).t() @ dy.double()
                        for k in range(125)])
    first = None
    for _ in range(3):
        (dw,) = torch.autograd.grad(pack.sparse_conv_3d(x, w).jdata, w, dy)
        got = dw.permute(4, 3, 2, 1, 0).reshape(125, cin, cout)
        assert float((got.double() - want).norm() / want.norm()) <= torch.finfo(dtype).eps / 2 + 2e-5
        # every offset by itself: a tile taken from the wrong buffer shows in one block of offsets
        err = (got.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1).clamp(min=1e-30)
        assert float(err.max()) <= torch.finfo(dtype).eps / 2 + 2e-5
        first = dw if first is None else first
        assert torch.equal(dw, first)
    fvdb._lib.load().check_device_errors(cuda_device)
