"""The prior grid's build at the sizes where its tiles and runs end: grids smaller than a 32 x 8 patch plus the flood's step,
odd extents, and the prefix array from the occupied cells alone."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [(0.01, 0.01, 0.01), (0.4, 0.02, 1.3), (2.1, 0.9, 0.1), (3.05, 2.6, 1.9)])
def test_grid_against_the_oracle(extent):
    from livox_warp.mapgrid import PriorGrid

    rng = np.random.default_rng(int(100 * extent[0]) + 7)
    xyz = (rng.uniform(0.0, 1.0, (700, 3)) * extent - 0.3).astype(np.float32)
    nrm = rng.normal(0.0, 1.0, (700, 3)).astype(np.float32)
    host = PriorGrid.prepare({"xyz": xyz, "normal": nrm})
    grid = PriorGrid(host)
    grid.build()
    og = oracle.PriorGrid(oracle.prior_prepare(xyz, nrm))
    assert np.array_equal(grid.start.cpu().numpy(), host["start"])
    assert np.array_equal(grid.nn.cpu().numpy(), og.nn)
    assert np.array_equal(grid.df.cpu().numpy(), og.df)
    # a map prepared without the occupied cells (a file written before they were kept) builds the same
    old = PriorGrid({k: v for k, v in host.items() if k not in ("cells", "first")})
    old.build()
    for a, b in ((old.start, grid.start), (old.nn, grid.nn), (old.df, grid.df), (old.xyzp, grid.xyzp)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("ncell,cells", [(1, [0]), (5, [2]), (1024, [0, 1023]), (1023, [1022]), (2049, [1023, 1024, 2048]),
                                         (5000, []), (100000, None)])
def test_prefix_from_occupied_cells(ncell, cells):
    from livox_warp import _lib

    rng = np.random.default_rng(3)
    cells = np.sort(rng.choice(ncell, 4000, replace=False)) if cells is None else np.array(cells, np.int64)
    counts = rng.integers(1, 9, len(cells))
    full = np.zeros(ncell, np.int64)
    full[cells] = counts
    want = np.concatenate([[0], np.cumsum(full)]).astype(np.int32)
    n = int(counts.sum())
    first = (np.cumsum(counts) - counts).astype(np.int32)
    d = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.int32)).cuda()  # noqa: E731
    c, f, out = d(cells), d(first), torch.full((ncell + 2,), -7, dtype=torch.int32, device="cuda")
    _lib.call("lw_prior_starts", _lib.ptr(c), _lib.ptr(f), len(cells), n, ncell, _lib.ptr(out), _lib.stream_ptr())
    got = out.cpu().numpy()
    assert np.array_equal(got[:ncell + 1], want) and got[-1] == -7
