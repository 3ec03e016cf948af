"""Bricks that many points share, against the oracle: a warp's lanes of one brick claim it once, and mark it once from eight on,
and every point adds its sums in one reduction, or by atomics where the sums are not aligned for one."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

V = 0.1
SENSOR = (0.5, -0.25, 1.5)


def _cloud(kind, n, rng):
    """Points of bricks 4 V wide, corners at whole multiples of 4 V."""
    if kind == "one":
        return rng.uniform(0.0, 4 * V, (n, 3))
    if kind == "two":  # by turns
        p = rng.uniform(0.0, 4 * V, (n, 3))
        p[1::2, 0] += 4 * V
        return p
    if kind == "runs":  # runs of 1 to 12 points of a brick: groups below, at and above the line within a warp
        brick = np.repeat(rng.integers(-6, 6, (n, 3)), rng.integers(1, 13, n), axis=0)[:n]
        return (brick + rng.uniform(0.0, 1.0, (n, 3))) * 4 * V
    if kind == "same":  # one point over and over
        return np.full((n, 3), 0.123)
    raise ValueError(kind)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("n", [1, 31, 33, 2001, 40_007])
@pytest.mark.parametrize("kind", ["one", "two", "runs", "same"])
def test_crowded_bricks(kind, n, aligned):
    from livox_warp import gpu
    from livox_warp.perception import Perception

    rng = np.random.default_rng(n)
    xyz = _cloud(kind, n, rng).astype(np.float32)
    gnd = (rng.uniform(size=n) < 0.3).astype(np.int32)  # lanes without a point of the clusters
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << 16)
    pipe.load_points(xyz)
    pipe.gnd[:n].copy_(torch.from_numpy(gnd))
    perc = Perception(pipe, cluster_slots=1 << 17)
    pipe.neighborhoods(3 * V, True, SENSOR)  # makes the buffers
    if not aligned:
        sums = torch.empty(4 * len(perc._t["node_slot"]) + 1, dtype=torch.int64, device="cuda")[1:]
        perc.cb.st_sum = sums.data_ptr()
        acc = torch.empty(4 * pipe._nb.cap + 1, dtype=torch.int64, device="cuda")[1:]
        pipe._nb.acc = acc.data_ptr()
        assert sums.data_ptr() % 16 == 8 and acc.data_ptr() % 16 == 8
        pipe.neighborhoods(3 * V, True, SENSOR)
    for got, want in zip((pipe.nbr, pipe.nrm, pipe.curv), oracle.neighborhoods(xyz, 3 * V, True, SENSOR)):
        assert np.array_equal(got[:n].cpu().numpy(), want)
    found = perc.cluster(voxel=V, connect=0.15, min_pts=2)
    cid, labels, clusters, _ = oracle.cluster(xyz, gnd, voxel=V, connect=0.15, min_pts=2)
    assert perc.cc_converged and len(found) == len(clusters)
    assert np.array_equal(pipe.cid[:n].cpu().numpy(), cid) and np.array_equal(perc.node_labels(), labels)
    for c, (cnt, cen, lo, hi) in zip(found, clusters):
        assert c["cnt"] == cnt and np.array_equal(c["cen"].astype(np.float32), cen)
        assert np.array_equal(c["lo"].astype(np.float32), lo) and np.array_equal(c["hi"].astype(np.float32), hi)
