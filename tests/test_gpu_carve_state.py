"""What Pipeline.carve may touch: the misses, and a workspace of its own."""

import pytest
import torch

from test_gpu_carve import VOXEL, _mapped

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mapped():
    return _mapped((0.0, 0.0, 0.0))


def _want(pipe, sx, sa, sf, every):
    """lw_carve's misses."""
    from livox_warp import _lib
    from livox_warp.gpu import C_ref

    stop = torch.zeros(len(sf), dtype=torch.float32, device="cuda")
    pipe.map_miss.zero_()
    _lib.call("lw_carve", _lib.ptr(sx), 3, _lib.ptr(sa), _lib.ptr(sf), None, len(sf), _lib.ptr(pipe.poses), every,
              1.0 / VOXEL, 40.0, 4096, C_ref(pipe.map_struct), _lib.ptr(stop), _lib.stream_ptr())
    want = pipe.map_miss.clone()
    assert int(want.sum()) > 0
    pipe.map_miss.zero_()
    return want


@pytest.mark.parametrize("every", [1, 3])
def test_carving_leaves_the_insertion_scratch_alone(mapped, every):
    """The batch counts and the points' slots are an insertion's, which may be under way on another stream: whatever they
    hold stays, and is not read."""
    pipe, (sx, sa, sf) = mapped
    want = _want(pipe, sx, sa, sf, every)
    count, slot = pipe._map_bcnt.clone(), pipe._slot.clone()
    pipe._map_bcnt.copy_(torch.arange(pipe.map_cap, dtype=torch.int32, device="cuda") % 5)
    pipe._slot.fill_(-7)
    held = [v.clone() for v in (pipe.map_keys, pipe.map_cnt, pipe.map_acc, pipe.map_last, pipe.map_first,
                                pipe._map_bcnt, pipe._map_lead, pipe.map_stats, pipe._slot)]
    try:
        pipe.carve(sx, sa, sf, len(sf), VOXEL, every=every)
        now = (pipe.map_keys, pipe.map_cnt, pipe.map_acc, pipe.map_last, pipe.map_first, pipe._map_bcnt,
               pipe._map_lead, pipe.map_stats, pipe._slot)
        assert all(torch.equal(a, b) for a, b in zip(now, held))
        assert torch.equal(pipe.map_miss, want)
        assert int(pipe._carve_marks.abs().sum()) == 0, "the workspace's marks are not clean"
    finally:
        pipe._map_bcnt.copy_(count)
        pipe._slot.copy_(slot)
        pipe.map_miss.zero_()
