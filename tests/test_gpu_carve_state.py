"""What Pipeline.carve may touch: the misses, and a workspace of its own."""

import threading

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


def test_carves_from_several_streams_and_threads_take_turns(mapped):
    """Four threads with a stream each, carving at the same time with different strides: every call counts what it counts
    alone."""
    pipe, (sx, sa, sf) = mapped
    strides, rounds = (1, 2, 3, 5), 12
    want = sum(_want(pipe, sx, sa, sf, e) for e in strides) * rounds
    torch.cuda.synchronize()
    start, failed = threading.Barrier(len(strides)), []

    def work(every):
        try:
            stream = torch.cuda.Stream()
            start.wait(10.0)
            with torch.cuda.stream(stream):
                for _ in range(rounds):
                    pipe.carve(sx, sa, sf, len(sf), VOXEL, every=every)
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(e,)) for e in strides]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    got = pipe.map_miss.clone()
    pipe.map_miss.zero_()
    assert torch.equal(got, want)
    assert int(pipe._carve_marks.abs().sum()) == 0


def test_a_captured_carve_counts_like_an_eager_one(mapped):
    pipe, (sx, sa, sf) = mapped
    want = _want(pipe, sx, sa, sf, 2)
    pipe.carve(sx, sa, sf, len(sf), VOXEL, every=2)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        pipe.carve(sx, sa, sf, len(sf), VOXEL, every=2)
    g.replay()
    pipe.carve(sx, sa, sf, len(sf), VOXEL, every=2)
    torch.cuda.synchronize()
    got = pipe.map_miss.clone()
    pipe.map_miss.zero_()
    assert torch.equal(got, 3 * want)


def test_the_stream_of_the_carve_before_may_be_gone(mapped):
    """A carve on a stream the caller made and has destroyed since, then one on another stream: nothing of the first
    stream is kept."""
    import ctypes

    from livox_warp import gpu

    pipe, (sx, sa, sf) = mapped
    want = _want(pipe, sx, sa, sf, 2)
    cudart = torch.cuda.cudart()
    raw = ctypes.c_void_p()
    assert int(cudart.cudaStreamCreate(ctypes.addressof(raw))) == 0
    stream = torch.cuda.ExternalStream(raw.value)
    assert gpu._foreign(stream) and not gpu._foreign(torch.cuda.Stream()) and not gpu._foreign(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        pipe.carve(sx, sa, sf, len(sf), VOXEL, every=2)
    stream.synchronize()
    del stream
    assert int(cudart.cudaStreamDestroy(raw.value)) == 0
    pipe.carve(sx, sa, sf, len(sf), VOXEL, every=2)
    torch.cuda.synchronize()
    got = pipe.map_miss.clone()
    pipe.map_miss.zero_()
    assert torch.equal(got, 2 * want)
