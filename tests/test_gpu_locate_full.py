"""A full batch of scans whose last tiles are part empty takes the search in sorted order in every tile size that the autotuner
tries and in the graph's: the workspace holds all its slots."""

import numpy as np
import pytest
import torch

from livox_warp import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def site():
    from livox_warp.mapgrid import PriorGrid

    sc = synth.box_room(3)
    xyz, nrm = synth.sample_surfaces(sc, 0.05, 0, jitter=0.002)
    g = PriorGrid({"xyz": xyz, "normal": nrm})
    g.build()
    return sc, g


@pytest.mark.parametrize("tile", [32, 64, 128, 256])
def test_a_full_batch_is_searched_in_sorted_order(site, tile):
    from livox_warp.localize import GlobalLocalizer, tiling

    sc, g = site
    k, n = 128, 1025  # one point over a multiple of every tile size; the two make the smallest batch there is, and a little
    T = np.repeat(synth.free_poses(sc, 1, 4, z=1.2, margin=0.4), k, axis=0)
    scan = synth.spin_scan(sc, T[0], n, 7)
    n = len(scan)
    loc = GlobalLocalizer(g, hyp_cap=k, pts_cap=k * n)
    b = loc.batch
    assert b.pts_cap == max(k * n, loc.PTS_CAP)
    pts = torch.zeros((k * n, 4), dtype=torch.float32)
    pts[:, :3] = torch.from_numpy(np.tile(scan, (k, 1)))
    hi = n * np.arange(1, k + 1)
    lo = hi - n
    slots = len(tiling(lo, hi, tile)[0]) * tile
    b.match.fill_(-7)
    got = loc.register_packed(pts, lo, hi, T, schedule=((0.3, 2),), tile=tile, blocks_per_sm=3)
    found = b.match[:slots].view(k, -1)[:, :n]
    assert int((found == -7).sum()) == 0, "the batch went the way without a workspace"
    assert np.array_equal(got.T, np.repeat(got.T[:1], k, axis=0)) and got.fit[0, 2] > 0.5
