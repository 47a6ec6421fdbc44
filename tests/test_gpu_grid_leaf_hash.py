"""Grids built through the leaf hash (2^18 rows and more) against the voxel sort that smaller inputs
take: the same voxels in the same order, offsets, bounding behaviour and leaf table, whole numbers
equal.  Repeated rows, empty grids, negative coordinates, several root tiles, voxels that fill a
leaf, more leaves than the table takes (the sort serves those), every point type."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

N = 1 << 18  # the rule's line


def _rows(kind, seed):
    """(ijk [n, 3], rows per grid)"""
    rng = np.random.default_rng(seed)
    if kind == "cloud":  # repeated hits, four grids of which one is empty
        sizes = [200000, 0, 150001, 3]
        parts = [rng.integers(-40, 40, (m, 3)) + 5 * i for i, m in enumerate(sizes)]
    elif kind == "tiles":  # clusters in different root tiles, both signs, up to the coordinate limit
        sizes = [N + 1]
        c = rng.choice([-(1 << 20), -4096, -8, 0, 4090, (1 << 20) - 30], (sizes[0], 3))
        parts = [c + rng.integers(0, 30, (sizes[0], 3))]
    elif kind == "full":  # one full leaf and a one-voxel leaf per grid
        sizes = [N // 2, N // 2]
        parts = [np.concatenate([rng.integers(0, 8, (m - 1, 3)), [[64, 0, 9]]]) for m in sizes]
    elif kind == "line":  # just below the line: the sort
        sizes = [N - 1]
        parts = [rng.integers(0, 64, (sizes[0], 3))]
    else:  # "sparse": about one row per leaf, beyond the table
        sizes = [N + 77]
        parts = [rng.integers(-3000, 3000, (sizes[0], 3))]
    return np.concatenate(parts).astype(np.int32), np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)


def _check(grid, ijk, off):
    import fvdb

    o_ijk, o_off = orc.grid_from_ijk(ijk, off)
    assert np.array_equal(grid.ijk.jdata.cpu().numpy(), o_ijk)
    assert np.array_equal(grid.joffsets.cpu().numpy(), o_off)
    assert np.array_equal(grid._impl.joffsets_host.numpy(), o_off)
    # the leaf table and lookups, against a grid of the unique voxels (the sort, where few enough)
    if o_ijk.shape[0] < N:
        dev = grid.ijk.jdata.device
        ref = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor.from_data_and_offsets(
            torch.from_numpy(o_ijk).to(dev), torch.from_numpy(o_off).to(dev)))
        assert torch.equal(grid._impl.leaves, ref._impl.leaves)
        assert torch.equal(grid.conv_grid(2, 2).ijk.jdata, ref.conv_grid(2, 2).ijk.jdata)
        q = grid.ijk_to_index(ref.ijk, cumulative=True).jdata
        assert torch.equal(q, torch.arange(o_ijk.shape[0], device=dev))


@pytest.mark.parametrize("kind", ["cloud", "tiles", "full", "line", "sparse"])
def test_ijk_rows(cuda_device, kind):
    import fvdb

    ijk, off = _rows(kind, 11)
    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor.from_data_and_offsets(
        torch.from_numpy(ijk).to(cuda_device), torch.from_numpy(off).to(cuda_device)))
    _check(grid, ijk, off)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["cloud", "full", "sparse"])
def test_points(cuda_device, kind, dtype):
    import fvdb

    ijk, off = _rows(kind, 12)
    ijk = np.clip(ijk, -900, 900)
    B = off.size - 1
    sizes = [[0.5 * (b + 1), 0.25, 2.0] for b in range(B)]
    orgs = [[0.5 * b, -1.0, 4.0] for b in range(B)]
    b = np.searchsorted(off, np.arange(ijk.shape[0]), side="right") - 1
    # powers of two and halves: every coordinate below is exact in 16 bits up to |ijk| of 128, and
    # the voxel a rounded point falls in is computed from the rounded point
    p = torch.from_numpy(ijk * np.asarray(sizes)[b] + np.asarray(orgs)[b]).to(dtype)
    acc = torch.float64 if dtype == torch.float64 else torch.float32
    s = torch.from_numpy(1.0 / np.asarray(sizes)[b]).to(acc)
    t = torch.from_numpy(-np.asarray(orgs)[b] / np.asarray(sizes)[b]).to(acc)
    want = torch.floor(torch.addcmul(t.double(), p.double(), s.double()) + 0.5).to(torch.int32).numpy()
    grid = fvdb.GridBatch.from_points(fvdb.JaggedTensor.from_data_and_offsets(
        p.to(cuda_device), torch.from_numpy(off).to(cuda_device)), sizes, orgs)
    _check(grid, want, off)


def test_out_of_range_rows_are_refused(cuda_device):
    import fvdb

    ijk, _ = _rows("cloud", 13)
    ijk[1234, 1] = 1 << 20
    with pytest.raises(ValueError):
        fvdb.GridBatch.from_ijk(torch.from_numpy(ijk).to(cuda_device))


@pytest.mark.parametrize("leaves", [511, 513, 65536, 65537])
def test_leaf_counts(cuda_device, leaves):
    """Edges of the leaf sort's tiles and its largest size (the radix sort serves more): distinct leaves
    in three grids, one of them empty, at least nine rows per leaf."""
    import fvdb

    rng = np.random.default_rng(leaves)
    n = max(N, 9 * leaves)
    side = 48
    cell = rng.permutation(side**3)[:leaves]
    origin = 8 * np.stack([cell // side**2 - 20, cell // side % side - 7, cell % side], 1)
    which = np.concatenate([np.arange(leaves), rng.integers(0, leaves, n - leaves)])
    ijk = (origin[which] + rng.integers(0, 8, (n, 3))).astype(np.int32)
    grid_of = np.sort(which % 2) * 2  # grids 0 and 2
    ijk = ijk[np.argsort(which % 2, kind="stable")]
    off = np.searchsorted(grid_of, np.arange(4)).astype(np.int64)
    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor.from_data_and_offsets(
        torch.from_numpy(ijk).to(cuda_device), torch.from_numpy(off).to(cuda_device)))
    assert grid._impl.total_leaf_nodes == leaves
    _check(grid, ijk, off)


@pytest.mark.parametrize("rows_per_leaf", [1.0, 5.0, 7.9, 8.1, 10.0])
def test_inputs_near_and_past_the_table_size(cuda_device, rows_per_leaf):
    """Rows in random order: the table overflows, or nearly, while every CTA is still inserting; the sort
    that takes over works inside the bounding box that the insertion measured."""
    import fvdb

    n = N + 70001
    leaves = int(n / rows_per_leaf)
    rng = np.random.default_rng(leaves)
    side = 80
    cell = rng.permutation(side**3)[:leaves]
    origin = 8 * np.stack([cell // side**2 - 60, cell // side % side - 33, cell % side + 11], 1)
    which = np.concatenate([np.arange(leaves), rng.integers(0, leaves, n - leaves)])
    ijk = (origin[rng.permutation(which)] + rng.integers(0, 8, (n, 3))).astype(np.int32)
    off = np.array([0, n // 3, n // 3, n], dtype=np.int64)
    grid = fvdb.GridBatch.from_ijk(fvdb.JaggedTensor.from_data_and_offsets(
        torch.from_numpy(ijk).to(cuda_device), torch.from_numpy(off).to(cuda_device)))
    _check(grid, ijk, off)
    # the coarse grid's keys cover the fine grid's box
    assert np.array_equal(grid.conv_grid(2, 2).ijk.jdata.cpu().numpy(), orc.grid_from_ijk(ijk >> 1, off)[0])


@pytest.mark.parametrize("at", [0, -1])
def test_out_of_range_rows_among_too_many_leaves_are_refused(cuda_device, at):
    import fvdb

    ijk = np.random.default_rng(5).integers(-(1 << 13), 1 << 13, (8 * N, 3)).astype(np.int32)
    ijk[at, 2] = -(1 << 20) - 1
    with pytest.raises(ValueError):
        fvdb.GridBatch.from_ijk(torch.from_numpy(ijk).to(cuda_device))
