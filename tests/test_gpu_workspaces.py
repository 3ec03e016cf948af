"""Workspaces hold what their passes use: bytes per table slot, per point and per sample."""

import pytest

pytestmark = pytest.mark.gpu


def _bytes(tensors):
    return sum(t.numel() * t.element_size() for t in tensors.values())


def test_neighbourhood_buffers():
    from livox_warp import gpu

    pipe = gpu.Pipeline(ring_capacity=1 << 14, map_capacity=1 << 14)
    pipe.neighborhoods(0.3, True, (0.0, 0.0, 0.0))
    # key 8, mask 8, first voxel 4; per voxel the sums 32, count 4, normal 12, curvature 4
    assert _bytes(pipe._nb_t) <= 72 * pipe._nb.cap + 4 * pipe._nb.pt_cap + 1024


def test_cluster_buffers():
    from livox_warp import gpu
    from livox_warp.perception import Perception

    pipe = gpu.Pipeline(ring_capacity=1 << 10, map_capacity=1 << 10)
    perc = Perception(pipe, cluster_slots=1 << 18)
    assert _bytes(perc._t) <= 40 * (1 << 18) + (1 << 19)  # a key and the masks, bases and labels in acc; points and clusters


def test_network_scratch():
    from livox_warp import initnet

    net = initnet.InitNet(seed=0, batch_cap=64)
    # per sample: two sets' 256 channels (gradient, place, a row of 128 bf16), sums of 8576 floats, and the head's vectors
    assert _bytes(net._scr) <= 64 * (2 * 256 * (4 + 4 + 256) + 2 * 8576 * 4 + (128 + 6 + 512 + 1) * 4) + 1024
