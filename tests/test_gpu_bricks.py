"""Neighbourhoods and clusters through bricks of 4 x 4 x 4 voxels, against the oracle, where the bricks' bookkeeping can go
wrong: one voxel per brick (32 bricks among 32 voxels), full bricks (64 voxels), one brick, one point, runs across
brick borders, negative coordinates, and the end of the voxel keys' range."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

V = 0.1


def _cloud(kind, rng):
    if kind == "sparse":  # voxels mostly alone in their brick
        return (rng.integers(-400, 400, (4000, 3)) * 0.2 * V + V * rng.uniform(0.1, 0.9, (4000, 3)))
    if kind == "chains":  # random walks of one voxel per step: long thin components through many bricks
        steps = np.cumsum(rng.integers(-1, 2, (40, 200, 3)), axis=1) + rng.integers(-60, 60, (40, 1, 3))
        return (steps.reshape(-1, 3) + rng.uniform(0.2, 0.8, (8000, 3))) * V
    if kind == "full":  # every voxel of a block of bricks
        g = np.stack(np.meshgrid(*[np.arange(-9, 15)] * 3, indexing="ij"), -1).reshape(-1, 3)
        return (g + rng.uniform(0.2, 0.8, g.shape)) * V
    if kind == "one":
        return np.array([[0.31, -0.17, 2.05]])
    if kind == "brick":
        return rng.uniform(0.41, 0.79, (300, 3))
    if kind == "edge":  # where the 21-bit fields of the key start again
        p = rng.uniform(-1.5, 1.5, (6000, 3))
        p[:, 0] += (1 << 20) * V
        return p
    if kind == "far":
        return rng.uniform(-2.0, 2.0, (6000, 3)) + (5210.0, -7300.0, 812.0)
    raise ValueError(kind)


KINDS = ("sparse", "chains", "full", "one", "brick", "edge", "far")


def _pipe(xyz):
    from livox_warp import gpu

    pipe = gpu.Pipeline(ring_capacity=1 << 15, map_capacity=1 << 15)
    pipe.load_points(xyz)
    return pipe


@pytest.mark.parametrize("connect", [0.09, 0.16, 0.31, 0.4])
@pytest.mark.parametrize("kind", KINDS)
def test_clusters(kind, connect):
    from livox_warp.perception import Perception

    xyz = _cloud(kind, np.random.default_rng(3)).astype(np.float32)
    pipe = _pipe(xyz)
    perc = Perception(pipe, cluster_slots=1 << 16)
    for _ in range(2):  # the second call finds what the first left in the buffers
        found = perc.cluster(voxel=V, connect=connect, min_pts=5, use_ground=False)
        cid = pipe.cid[:len(xyz)].cpu().numpy()
        ocid, olabels, oclusters, _ = oracle.cluster(xyz, None, voxel=V, connect=connect, min_pts=5)
        assert perc.cc_converged
        assert np.array_equal(perc.node_labels(), olabels)
        assert np.array_equal(cid, ocid)
        assert len(found) == len(oclusters)
        for c, (cnt, cen, lo, hi) in zip(found, oclusters):
            assert c["cnt"] == cnt
            assert np.array_equal(c["cen"].astype(np.float32), cen)
            assert np.array_equal(c["lo"].astype(np.float32), lo) and np.array_equal(c["hi"].astype(np.float32), hi)


@pytest.mark.parametrize("radius", [0.05, 0.3, 2.5])
@pytest.mark.parametrize("kind", KINDS)
def test_neighbourhoods(kind, radius):
    xyz = _cloud(kind, np.random.default_rng(4)).astype(np.float32)
    pipe = _pipe(xyz)
    sensor = (0.5, -0.25, 1.5)
    pipe.neighborhoods(radius, True, sensor)
    n = len(xyz)
    cnt, nrm, curv = oracle.neighborhoods(xyz, radius, True, sensor)
    assert np.array_equal(pipe.nbr[:n].cpu().numpy(), cnt)
    assert np.array_equal(pipe.nrm[:n].cpu().numpy(), nrm) and np.array_equal(pipe.curv[:n].cpu().numpy(), curv)


def test_a_table_too_small_reads_as_crowded():
    """With room for 1024 bricks and 4000 lone voxels, the points that found none read as crowded, flat and facing up,
    and the others as in a table of their own."""
    from livox_warp import _lib

    xyz = _cloud("sparse", np.random.default_rng(5)).astype(np.float32)
    pipe = _pipe(xyz)
    n = len(xyz)
    pipe.neighborhoods(0.3, True, (0.0, 0.0, 0.0))
    want = [pipe.nbr[:n].clone(), pipe.nrm[:n].clone(), pipe.curv[:n].clone()]
    t = pipe._nb_t
    small = _lib.NbrBuf(*(_lib.ptr(t[k]).value for k in _lib.NbrBuf.PTRS), 1024, pipe.work_cap)
    sen = (_lib.f32 * 3)(0.0, 0.0, 0.0)
    import ctypes

    _lib.call("lw_neighborhoods", _lib.ptr(pipe.c_xyz), 3, None, n, 0.3, 1, sen, ctypes.byref(small),
              _lib.ptr(pipe.nbr), _lib.ptr(pipe.nrm), _lib.ptr(pipe.curv), _lib.stream_ptr())
    torch.cuda.synchronize()
    lost = pipe.nbr[:n] == 1 << 30
    assert 0 < int(lost.sum()) < n
    assert bool((pipe.nrm[:n][lost] == torch.tensor([0.0, 0.0, 1.0], device="cuda")).all())
    assert bool((pipe.curv[:n][lost] == 0).all())
    assert bool((pipe.nbr[:n][~lost] <= want[0][~lost]).all())
