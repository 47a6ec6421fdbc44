"""What run_alone hands back is the caller's to keep: ordinary host memory with contents of its own."""

import pytest
import torch

from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [(3000, 2999), (60000, 59999)])  # below and above the size that is staged
def test_results_are_ordinary_memory(cuda_device, rows):
    import fvdb
    from fvdb.serving import ConvStack, Request, run_alone

    g = torch.Generator().manual_seed(1)
    ijk = [torch.from_numpy(random_sparse_ijk(n, 60, n)) for n in rows]
    reqs = [Request(i, v, torch.randn(v.shape[0], 16, generator=g).bfloat16()) for i, v in enumerate(ijk)]
    model = ConvStack([16, 32, 24], cuda_device)
    first = [run_alone(model, r, cuda_device) for r in reqs]
    again = [run_alone(model, r, cuda_device) for r in reqs]  # may reuse whatever the first calls released
    for (y, v), (y2, v2), r in zip(first, again, reqs):
        assert y.device.type == v.device.type == "cpu" and not y.is_pinned() and not v.is_pinned()
        assert torch.equal(y, y2) and torch.equal(v, v2)
        grid = fvdb.GridBatch.from_ijk(r.ijk.to(cuda_device))
        assert torch.equal(v, grid.ijk.jdata.cpu())
        x = torch.zeros(grid.total_voxels, 16, dtype=torch.bfloat16, device=cuda_device)
        x[grid.ijk_to_index(r.ijk.to(cuda_device), cumulative=True).jdata] = r.features.to(cuda_device)
        assert torch.equal(y, model(grid, x).cpu())
