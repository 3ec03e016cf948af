"""lw_carve_ws (planes fitted once per voxel met, pairs tested afterwards) counts the misses lw_carve counts, bit for
bit, also where its lists are full, where few rays leave warps part empty and where nothing is met."""

import ctypes

import numpy as np
import pytest
import torch

import common

pytestmark = pytest.mark.gpu

VOXEL = 0.1


def _mapped(origin):
    """A map of five frames of the handheld path (moved by `origin`), and a sixth frame to carve with from a pose some
    way off, so that its rays cross what the map holds."""
    from livox_warp import gpu

    traj = common.handheld()
    frames = common.handheld_frames(16)[10:16]
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << 18)
    view = gpu.make_view(now=1.6, voxel=VOXEL, map_cap=pipe.map_cap)
    for j, (x, a, t) in enumerate(frames):
        T = common.mid_pose(traj, 10 + j)
        T[:3, 3] += origin
        pipe.set_pose(10 + j, T.astype(np.float32))
        sx, sa, st, sf = pipe.stage(x, a, t, len(t), 10.0)
        if j < 5:
            pipe.map_insert(sx, sa, st, sf, len(t), view, VOXEL)
    T[:3, 3] += (0.4, -0.3, -0.3)
    pipe.set_pose(15, T.astype(np.float32) @ gpu.mount_matrix(0.0, 4.0, 6.0, 0.0, 0.0, 0.0))
    pipe.flush_poses()
    return pipe, [v[:len(t)].clone() for v in (sx, sa, sf)]


@pytest.fixture(scope="module")
def mapped():
    return _mapped((0.0, 0.0, 0.0))


def _misses(pipe, call):
    from livox_warp import _lib

    pipe.map_miss.zero_()
    call(_lib)
    torch.cuda.synchronize()
    assert int(pipe._map_bcnt.abs().sum()) == 0, "the map's scratch is not clean"
    return pipe.map_miss.clone()


@pytest.mark.parametrize("n,every,max_steps,pairs,slots", [
    (10000, 1, 4096, 1 << 18, 1 << 16),  # roomy
    (10000, 2, 4096, 1 << 18, 7),        # few voxels fit the list: the pair pass fits the others
    (10000, 3, 4096, 100, 1 << 16),      # few pairs fit: the walk tests the others
    (9973, 1, 4096, 0, 0),               # no workspace at all
    (10000, 1, 65, 1 << 18, 1 << 16),    # cut short just past two rounds of 32 steps
    (1, 1, 4096, 64, 64),                # one ray
    (35, 4, 4096, 64, 64),               # nine rays: the last warp holds one
    (9999, 20000, 4096, 64, 64),         # one ray of many points
])
def test_workspace_carving_counts_the_same_misses(mapped, n, every, max_steps, pairs, slots):
    _compare(mapped, n, every, max_steps, pairs, slots)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_keys_wrap_where_the_voxel_range_ends(axis):
    """Rays that cross the 2^20th voxel of an axis, where the key's 21-bit field starts again at zero."""
    origin = np.zeros(3)
    origin[axis] = (1 << 20) * VOXEL - (3.0, 3.0, 1.0)[axis]
    _compare(_mapped(origin), 10000, 1, 4096, 1 << 18, 1 << 16)


def _compare(mapped, n, every, max_steps, pairs, slots):
    from livox_warp.gpu import C_ref

    pipe, (sx, sa, sf) = mapped
    n = min(n, len(sf))
    stop = torch.zeros(max(n, 1), dtype=torch.float32, device="cuda")
    bufs = (torch.empty(max(pairs, 1), dtype=torch.int64, device="cuda"),
            torch.empty(max(pairs, 1), dtype=torch.float32, device="cuda"),
            torch.empty((max(slots, 1), 8), dtype=torch.float32, device="cuda"),
            torch.empty(max(slots, 1), dtype=torch.int32, device="cuda"),
            torch.full((3,), 99, dtype=torch.int64, device="cuda"))

    def args(_lib):
        return (_lib.ptr(sx), 3, _lib.ptr(sa), _lib.ptr(sf), None, n, _lib.ptr(pipe.poses), every, 1.0 / VOXEL, 40.0,
                max_steps, C_ref(pipe.map_struct), _lib.ptr(stop))

    def old(_lib):
        _lib.call("lw_carve", *args(_lib), _lib.stream_ptr())

    def new(_lib):
        ws = _lib.CarveBuf(*(_lib.ptr(b) for b in bufs), pairs, slots)
        _lib.call("lw_carve_ws", *args(_lib), ctypes.byref(ws), _lib.stream_ptr())

    want, got = _misses(pipe, old), _misses(pipe, new)
    assert torch.equal(want, got)
    if n > 1000 and every < 10 and max_steps > 1000:
        assert int(want.sum()) > 0, "no ray pierced anything: the test is vacuous"
