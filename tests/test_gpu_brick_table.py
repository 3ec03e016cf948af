"""The table of the neighbourhoods' and clusters' bricks where every brick holds one voxel, so that it is as full as it
gets: no point may be lost to a full probe window, whatever the order the points come in. Against the oracle."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

RADIUS, MAP_VOXEL = 0.1, 0.15  # a viewer's usual radius over a usual map: lone voxels in bricks of 4/3 of the radius
SENSOR = (0.5, -0.25, 1.5)


def _hall(width, depth, height, seed):
    """One point somewhere in every map voxel of the floor, the ceiling and the walls of a hall, float32."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = int(width / MAP_VOXEL), int(depth / MAP_VOXEL), int(height / MAP_VOXEL)
    faces = []
    for axis, far in ((2, nz), (1, ny), (0, nx)):
        dims = [nx, ny, nz]
        for at in (0, far):
            spans = [np.arange(d) for d in dims]
            spans[axis] = np.array([at])
            faces.append(np.stack(np.meshgrid(*spans, indexing="ij"), -1).reshape(-1, 3))
    ijk = np.unique(np.concatenate(faces), axis=0)
    return ((ijk + rng.uniform(0.05, 0.95, ijk.shape)) * MAP_VOXEL).astype(np.float32)


def _same_home(count, slots, cell):
    """Centres of `count` voxels, each alone in its brick, whose brick keys a multiplication by the golden ratio puts in the
    same slot of `slots`: they fill any window that starts there."""
    i, j = np.meshgrid(np.arange(2000), np.arange(2000), indexing="ij")
    half = (1 << 20) >> 2
    key = (i.reshape(-1).astype(np.uint64) + np.uint64(half)) | ((j.reshape(-1).astype(np.uint64) + np.uint64(half))
                                                                << np.uint64(19)) | (np.uint64(half) << np.uint64(38))
    with np.errstate(over="ignore"):
        h = (key * np.uint64(0x9E3779B97F4A7C15)).view(np.int64)
    home = (h ^ (h >> 29)) & (slots - 1)
    pick = np.flatnonzero(home == home[0])[:count]
    assert len(pick) == count
    ij = np.stack([i.reshape(-1)[pick], j.reshape(-1)[pick], np.zeros(count, np.int64)], -1)
    return ((4 * ij + 1.5) * cell).astype(np.float32)


def _pipe(xyz):
    from livox_warp import gpu

    cap = max(1 << 16, 1 << (len(xyz) - 1).bit_length())
    pipe = gpu.Pipeline(ring_capacity=cap, map_capacity=cap)
    pipe.load_points(xyz)
    return pipe


def _neighbourhoods(pipe, xyz, radius):
    pipe.load_points(xyz)
    pipe.neighborhoods(radius, True, SENSOR)
    n = len(xyz)
    return [v[:n].cpu().numpy() for v in (pipe.nbr, pipe.nrm, pipe.curv)]


CLOUDS = {
    "hall": lambda: _hall(110.0, 88.0, 6.0, 1),  # just under 2^20 points, the fullest a table gets
    "corridors": lambda: _hall(60.0, 40.0, 3.0, 2),
    "one home": lambda: _same_home(300, 1024, RADIUS / 3.0),
}


@pytest.mark.parametrize("kind", CLOUDS)
def test_lone_voxels_keep_their_neighbourhoods(kind):
    xyz = CLOUDS[kind]()
    pipe = _pipe(xyz)
    got = _neighbourhoods(pipe, xyz, RADIUS)
    assert not (got[0] == 1 << 30).any(), "points lost to a full window"
    for g, w in zip(got, oracle.neighborhoods(xyz, RADIUS, True, SENSOR)):
        assert np.array_equal(g, w)
    for seed in (3, 4):  # other orders of arrival
        p = np.random.default_rng(seed).permutation(len(xyz))
        for a, b in zip(_neighbourhoods(pipe, xyz[p], RADIUS), got):
            assert np.array_equal(a, b[p])


@pytest.mark.parametrize("kind", ["corridors", "one home"])
def test_lone_voxels_keep_their_cluster(kind):
    from livox_warp.perception import Perception

    xyz = CLOUDS[kind]()
    cell = RADIUS / 3.0
    pipe = _pipe(xyz)
    perc = Perception(pipe, cluster_slots=max(1 << 10, 1 << (2 * len(xyz) - 1).bit_length()))
    perc.cluster(voxel=cell, connect=3.9 * cell, min_pts=1, use_ground=False)
    _, labels, _, _ = oracle.cluster(xyz, None, voxel=cell, connect=3.9 * cell, min_pts=1)
    assert perc.cc_converged
    got = perc.node_labels()
    assert len(got) == len(labels), "points lost to a full window"
    assert np.array_equal(got, labels)


def test_points_that_found_room_are_as_if_the_others_were_not_there():
    """A table far too small (room for 1024 of some 4,000 bricks): what is lost is reported as crowded, flat and facing up;
    the rest have the neighbourhoods of the points that found room."""
    import ctypes

    from livox_warp import _lib

    rng = np.random.default_rng(5)
    xyz = (rng.integers(-400, 400, (4000, 3)) * 0.02 + rng.uniform(0.002, 0.018, (4000, 3))).astype(np.float32)
    pipe = _pipe(xyz)
    pipe.neighborhoods(0.3, True, SENSOR)  # makes the buffers
    t, n = pipe._nb_t, len(xyz)
    small = _lib.NbrBuf(*(_lib.ptr(t[k]).value for k in _lib.NbrBuf.PTRS), 1024, pipe.work_cap)
    _lib.call("lw_neighborhoods", _lib.ptr(pipe.c_xyz), 3, None, n, 0.3, 1, (_lib.f32 * 3)(*SENSOR),
              ctypes.byref(small), _lib.ptr(pipe.nbr), _lib.ptr(pipe.nrm), _lib.ptr(pipe.curv), _lib.stream_ptr())
    torch.cuda.synchronize()
    got = [v[:n].cpu().numpy() for v in (pipe.nbr, pipe.nrm, pipe.curv)]
    lost = got[0] == 1 << 30
    assert 0 < lost.sum() < n
    for g, w in zip(got, oracle.neighborhoods(xyz[~lost], 0.3, True, SENSOR)):
        assert np.array_equal(g[~lost], w)
