"""pbf_cell_sort_noalloc at the table sizes where its scan changes form (a
cluster holding 1 to 18 cells a thread, three kernels beyond), with and
without particles: permutation and ranges of a stable sort by cell."""
import numpy as np
import pytest

from ssf_pbf_cuda_gb300 import api
from tests.test_zz_no_alloc import noalloc_sort

pytestmark = pytest.mark.gpu

GRIDS = [(1, 1, 1), (32, 32, 16), (32, 32, 32), (64, 32, 32), (64, 64, 32), (64, 64, 64), (128, 64, 64)]


@pytest.mark.parametrize("n", [0, 1, 5000])
@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
def test_noalloc_sort_by_table_size(gpu, grid, n):
    rng = np.random.default_rng(n + grid[0])
    x = (rng.uniform(0.0, 1.0, size=(n, 3)) * np.array(grid) * 0.25).astype(np.float32)
    perm, start, end = noalloc_sort(api.load(), x, grid, 0.25)
    c = np.floor(x / np.float32(0.25)).astype(np.int64) % np.array(grid)
    key = (c[:, 2] * grid[1] + c[:, 1]) * grid[0] + c[:, 0]
    want = np.argsort(key, kind="stable")
    b = np.searchsorted(key[want], np.arange(int(np.prod(grid)) + 1))
    none = b[1:] == b[:-1]
    assert np.array_equal(perm, want.astype(np.uint32))
    assert np.array_equal(start, np.where(none, 0xFFFFFFFF, b[:-1]).astype(np.uint32))
    assert np.array_equal(end, np.where(none, 0xFFFFFFFF, b[1:]).astype(np.uint32))
