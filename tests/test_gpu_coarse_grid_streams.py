"""Coarse grids are built on a stream of the library's own and completed at their first use: the
buffers that the build reads and writes stay theirs meanwhile -- the fine grid's after the caller has
dropped it, the coarse grid's own on every stream that the caller may use it on."""

import numpy as np
import pytest
import torch

from tests.helpers import random_sparse_ijk

pytestmark = pytest.mark.gpu


def _fine(fvdb, dev, n, extent, seed):
    return fvdb.GridBatch.from_ijk(torch.from_numpy(random_sparse_ijk(n, extent, seed)).to(dev))


# 20,000 voxels in 2,197 leaves build through the hash, 60,000 in as many leaves through the sort
@pytest.mark.parametrize("n,extent", [(20000, 104), (60000, 1024)])
def test_the_fine_grid_may_be_dropped_before_the_coarse_grid_is_used(cuda_device, n, extent):
    import fvdb

    ijk = random_sparse_ijk(n, extent, 3)
    fine = _fine(fvdb, cuda_device, n, extent, 3)
    at = fine.ijk.jdata.data_ptr()
    shape = fine.ijk.jdata.shape
    coarse = fine.conv_grid(2, 2)
    del fine
    # what the caller allocates and overwrites next must not be the fine grid's memory
    taken = [torch.full(shape, -1, dtype=torch.int32, device=cuda_device) for _ in range(4)]
    assert at not in [t.data_ptr() for t in taken]
    want = np.unique(ijk // 2, axis=0)
    got = np.unique(coarse.ijk.jdata.cpu().numpy(), axis=0)
    assert coarse.total_voxels == want.shape[0] and np.array_equal(got, want)


def test_a_coarse_grid_completed_on_another_stream_stays_with_its_callers_stream(cuda_device):
    import fvdb

    fine = _fine(fvdb, cuda_device, 20000, 104, 4)
    other = torch.cuda.Stream(device=cuda_device)
    caller = torch.cuda.current_stream(cuda_device)
    coarse = fine.conv_grid(2, 2)
    with torch.cuda.stream(other):
        coarse.total_voxels  # completes the grid
    at = coarse.ijk.jdata.data_ptr()
    want = coarse.ijk.jdata.cpu()
    torch.cuda._sleep(400_000_000)  # about 0.2 s of the caller's stream, then a read of the grid
    got = coarse.ijk.jdata.clone()
    del coarse
    again = fine.conv_grid(4, 4)
    with torch.cuda.stream(other):
        again.total_voxels
    busy = not caller.query()
    assert busy and again.ijk.jdata.data_ptr() != at
    assert torch.equal(got.cpu(), want)
