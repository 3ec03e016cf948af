"""The batched registration with a workspace (nearest points found in sorted order, each from its last match) gives the poses,
counts, fits and iteration count of the one without, bit for bit: scans of uneven length, one shared scan, starts near
and far (queries beyond one cell, beyond the band and outside the grid), a workspace too small, and an empty schedule."""

import numpy as np
import pytest
import torch

from livox_warp import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    from livox_warp.mapgrid import PriorGrid

    sc = synth.box_room(3)
    xyz, nrm = synth.sample_surfaces(sc, 0.03, 0, jitter=0.002)
    g = PriorGrid({"xyz": xyz, "normal": nrm})
    g.build()
    return sc, g


def _both(loc, run):
    """run() with the workspace, then without."""
    from livox_warp import _lib

    got = run()
    keep = loc.batch.ws
    loc.batch.ws = _lib.LocWs(None, None, 0)
    want = run()
    loc.batch.ws = keep
    assert np.array_equal(got.T, want.T) and np.array_equal(got.count, want.count)
    assert np.array_equal(got.fit, want.fit) and got.iters == want.iters
    return got


@pytest.mark.parametrize("tile,ctas", [(32, 5), (64, 3), (128, 2), (32, 6), (96, 4)])
@pytest.mark.parametrize("shift", [0.05, 0.6, 4.0, 60.0])
def test_same_results(grid, tile, ctas, shift):
    from livox_warp.localize import GlobalLocalizer

    sc, g = grid
    rng = np.random.default_rng(int(10 * shift) + tile)
    true = synth.free_poses(sc, 7, 5, z=1.2, margin=0.4)
    scans = [synth.spin_scan(sc, true[h], n, 50 + h) for h, n in enumerate((1, 31, 33, 400, 2500, 129, 1000))]
    T0 = np.array(true)
    T0[:, :3, 3] += rng.uniform(-shift, shift, (7, 3))
    loc = GlobalLocalizer(g, hyp_cap=8, pts_cap=1 << 13)
    _both(loc, lambda: loc.register_batch(scans, T0, tile=tile, blocks_per_sm=ctas))
    _both(loc, lambda: loc.register_batch(scans, T0, schedule=(), tile=tile, blocks_per_sm=ctas))
    _both(loc, lambda: loc.register_batch(scans, T0, schedule=((0.2, 1),), tile=tile, blocks_per_sm=ctas))


def test_shared_scan_and_small_workspace(grid):
    """All poses on one scan (as icp() and refine() have it), and more tiles than the workspace holds."""
    from livox_warp import _lib
    from livox_warp.localize import SCHEDULE_ICP, GlobalLocalizer

    sc, g = grid
    true = synth.free_poses(sc, 1, 6, z=1.2, margin=0.4)
    scan = synth.spin_scan(sc, true[0], 3000, 9)
    T0 = synth.perturb(np.repeat(true, 5, axis=0), 3, 0.2, 3.0)
    loc = GlobalLocalizer(g, hyp_cap=8, pts_cap=1 << 14)
    s = torch.cuda.current_stream()
    loc._upload_pts([scan], s)
    n = len(scan)
    run = lambda: loc._run(np.zeros(5, np.int64), np.full(5, n, np.int64), T0, SCHEDULE_ICP, s, 32, 5)  # noqa: E731
    want = _both(loc, run)
    loc.batch.ws = _lib.LocWs(loc.batch.ws.sorted, loc.batch.ws.match, 5 * n)  # short of the last tile's rounding
    got = run()
    assert np.array_equal(got.T, want.T) and np.array_equal(got.fit, want.fit)
