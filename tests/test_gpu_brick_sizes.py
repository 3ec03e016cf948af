"""Neighbourhoods and clusters around the point counts where CTAs change from 8 to 32 voxels and the warps that sum up
clusters from one round of nodes to several, against the oracle."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

V = 0.1


def _points(n, rng):
    """Lone voxels, a few dense boxes and a long wall: bricks of one voxel up to 64, components small and large."""
    parts = [rng.uniform(-40.0, 40.0, (n // 3, 3)), rng.uniform(0.0, 2.0, (n // 3, 3)) + (3.0, -1.0, 0.4)]
    m = n - sum(len(p) for p in parts)
    parts.append(np.stack([rng.uniform(-20.0, 20.0, m), np.full(m, 5.03) + rng.normal(0.0, 0.02, m),
                           rng.uniform(0.0, 3.0, m)], -1))
    return rng.permutation(np.concatenate(parts)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 7, 9, 33, "line", "line + 1", "line + 8", 20001, 60003])
def test_sizes(n):
    from livox_warp import gpu
    from livox_warp.perception import Perception

    line = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    n = line + int(n[4:].replace(" ", "") or 0) if isinstance(n, str) else n
    xyz = _points(n, np.random.default_rng(n))
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << 16)
    pipe.load_points(xyz)
    sensor = (0.5, -0.25, 1.5)
    pipe.neighborhoods(0.3, True, sensor)
    for got, want in zip((pipe.nbr, pipe.nrm, pipe.curv), oracle.neighborhoods(xyz, 0.3, True, sensor)):
        assert np.array_equal(got[:n].cpu().numpy(), want)
    perc = Perception(pipe, cluster_slots=1 << 18)
    found = perc.cluster(voxel=V, connect=0.25, min_pts=3, use_ground=False)
    cid, labels, clusters, _ = oracle.cluster(xyz, None, voxel=V, connect=0.25, min_pts=3)
    assert perc.cc_converged and len(found) == len(clusters)
    assert np.array_equal(perc.node_labels(), labels) and np.array_equal(pipe.cid[:n].cpu().numpy(), cid)
    for c, (cnt, cen, lo, hi) in zip(found, clusters):
        assert c["cnt"] == cnt and np.array_equal(c["cen"].astype(np.float32), cen)
        assert np.array_equal(c["lo"].astype(np.float32), lo) and np.array_equal(c["hi"].astype(np.float32), hi)
