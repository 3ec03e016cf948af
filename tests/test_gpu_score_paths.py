"""lw_score_grid's two ways through a warp -- the table of (y, z) rows and the work per thread -- give every hypothesis the
same score: the scores are whole-number sums of the same float32 cells, so equal."""

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N_YAW, YAW0, DYAW = 12, 0.05, math.radians(30.0)


@pytest.fixture(scope="module")
def grid():
    from livox_warp import synth
    from livox_warp.mapgrid import PriorGrid

    xyz, nrm = synth.sample_surfaces(synth.box_room(3), 0.03, 0, jitter=0.002)
    grid = PriorGrid(PriorGrid.prepare({"xyz": xyz, "normal": nrm, "planarity": np.ones(len(xyz), np.float32)}))
    grid.build()
    return grid


def _score(grid, pts, pos, stride, tau=25.0):
    from livox_warp.localize import score_grid

    out = torch.full((len(pos) * N_YAW,), 7.0, dtype=torch.float32, device="cuda")
    score_grid(grid, torch.from_numpy(pts).cuda(), torch.from_numpy(pos).cuda(), N_YAW, YAW0, DYAW, tau, 10.0, out,
               pos_stride=stride)
    return out.cpu().numpy().reshape(len(pos), N_YAW)


def _points(n, seed):
    return np.random.default_rng(seed).uniform(-4.0, 4.0, (n, 3)).astype(np.float32) * np.float32([1, 1, 0.3])


@pytest.mark.parametrize("n_pts", [0, 1, 15, 17, 1024, 1025])
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 5), (64, 2), (65, 3), (7, 40)])  # rows a warp: one, many, straddled
def test_rows_and_list_order_agree(grid, n_pts, nx, ny):
    lo, hi = np.asarray(grid.lo), np.asarray(grid.hi)
    x = np.linspace(lo[0] - 0.2, hi[0] + 0.2, nx)
    y = np.linspace(lo[1] + 0.3, hi[1] - 0.3, ny)
    z = [lo[2] + 0.7, lo[2] + 1.3]
    pos = np.array([(a, b, c) for c in z for a in x for b in y], np.float32)
    pts = _points(n_pts, n_pts)
    rng = np.random.default_rng(nx)
    if nx > 1:
        pos[:2] = [[2.0, 2.0, 1.2], [2.2, 2.0, 1.2]]  # free whatever the spacing
    pos = np.concatenate([pos, pos[rng.permutation(len(pos))[:len(pos) // 2]]])  # the last ones out of order
    want = _score(grid, pts, pos, 1)
    assert nx == 1 or n_pts < 15 or (want > 0.0).any()
    shuffled = rng.permutation(len(pos))
    assert np.array_equal(_score(grid, pts, pos[shuffled], 1), want[shuffled])
    for stride in (ny, 2, len(pos), len(pos) + 9):
        assert np.array_equal(_score(grid, pts, pos, stride), want)


@pytest.mark.parametrize("tau", [0.5, 25.0, 1e6])
def test_points_far_away_or_not_finite(grid, tau):
    """Points far outside count nothing, whichever way a chunk goes: one point that is not finite sends its chunk the other
    way, and the finite points' sums stay what they are."""
    lo, hi = np.asarray(grid.lo), np.asarray(grid.hi)
    pos = np.array([(a, lo[1] + 2.0, lo[2] + 1.0) for a in np.linspace(lo[0], hi[0], 70)], np.float32)
    pts = _points(600, 5)
    want = _score(grid, pts, pos, 1, tau)
    assert (want > 0.0).any() and (want == -1.0).any()
    far = pts.copy()
    far = np.concatenate([far, np.float32([[1e6, 0, 0], [-1e9, 1e9, 0], [3e17, -3e17, 1e17], [0, 0, 1e12]])])
    assert np.array_equal(_score(grid, far, pos, 1, tau), want)
    for bad in (np.inf, -np.inf, 3e38):  # no cell: their rows lie outside the grid
        odd = np.concatenate([far, np.float32([[0.0, 0.0, bad]])])
        assert np.array_equal(_score(grid, odd, pos, 1, tau), want)
