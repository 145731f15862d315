"""pbf_cell_sort_noalloc with crowded cells: averages on both sides of the one
from which the rank is launched plainly (48 a cell), and buckets on both sides
of the sizes from which their members are read one by one (1,024) and sorted
by a block (4,096).  A stable sort by cell."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api
from tests.test_zz_no_alloc import noalloc_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,buckets", [
    ((2, 2, 2), [1023, 1024, 1025, 1, 0, 4096, 4097, 3]), ((4, 2, 2), [47] * 16), ((4, 2, 2), [48] * 16),
    ((1, 1, 1), [48]), ((8, 8, 8), [1025] + [40] * 511)], ids=["edges", "47", "48", "one", "mixed"])
def test_crowded_cells(gpu, grid, buckets):
    rng = np.random.default_rng(len(buckets))
    cell = np.repeat(np.arange(len(buckets)), buckets)
    cell = cell[rng.permutation(len(cell))]
    at = np.stack([cell % grid[0], cell // grid[0] % grid[1], cell // (grid[0] * grid[1])], 1)
    x = ((at + rng.uniform(0.1, 0.9, size=at.shape)) * 0.25).astype(np.float32)
    for _ in range(2):
        perm, start, end = noalloc_sort(api.load(), x, grid, 0.25)
        want = np.argsort(cell, kind="stable")
        b = np.concatenate([[0], np.cumsum(buckets)])
        none = np.asarray(buckets) == 0
        assert np.array_equal(perm, want.astype(np.uint32))
        assert np.array_equal(start, np.where(none, 0xFFFFFFFF, b[:-1]).astype(np.uint32))
        assert np.array_equal(end, np.where(none, 0xFFFFFFFF, b[1:]).astype(np.uint32))
