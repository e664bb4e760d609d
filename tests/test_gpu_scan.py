"""The prefix sum at the edges of its tiles of 8,192 elements, through the cell
sort on grids of one to three tiles: cell offsets, and the particles of each
cell in chain order (last inserted first), equal numpy's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 8191, 8192, 8193, 16384, 16385])
def test_cell_offsets_at_tile_edges(cells):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mps_b200 import _lib
    g = _lib.MpsGrid()
    g.dim = 2
    g.cell_size = 1.0
    g.dims[0], g.dims[1] = cells, 1
    n = 3 * cells + 5
    rng = np.random.default_rng(cells)
    cell = np.concatenate([rng.integers(0, cells, n - 2), [0, cells - 1]]).astype(np.int32)
    pos = torch.tensor(np.stack([cell + 0.5, np.full(n, 0.5)], 1).ravel(), device="cuda")
    typ = torch.zeros(n, dtype=torch.int32, device="cuda")
    out = [torch.full((k,), -7, dtype=torch.int32, device="cuda") for k in (n, n, cells + 1)]
    rc = _lib.load().mps_cell_sort_noalloc(C.byref(g), pos.data_ptr(), typ.data_ptr(), n, *(t.data_ptr() for t in out),
                                           torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0
    got_cell, order, start = (t.cpu().numpy() for t in out)
    assert np.array_equal(got_cell, cell)
    assert np.array_equal(start, np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=cells))]))
    assert np.array_equal(order, np.lexsort((-np.arange(n), cell)))


@pytest.mark.parametrize("cells", [10239, 10240, 10241])
def test_cell_offsets_at_long_tile_edges(cells):
    """Scans above 8,192 elements go by tiles of 2,048."""
    test_cell_offsets_at_tile_edges(cells)
