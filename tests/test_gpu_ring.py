"""The ring append and the frame copy against the indexed copies that they replace: whole values, so equal."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from livox_warp import _lib, gpu  # noqa: E402


def _batch(n, width, form, seed):
    g = torch.Generator().manual_seed(seed)
    wide = torch.randn((n + 3, 4), generator=g).cuda()
    if form == "rows":
        xyz = wide[:, :width].contiguous()
    elif form == "view":  # x, y, z of rows 4 floats apart
        xyz = wide[:, :3]
    elif form == "shifted":  # rows of 4 floats that start off a 16-byte boundary
        xyz = wide.reshape(-1)[1:1 + 4 * (n + 2)].view(n + 2, 4)
    else:  # "columns": columns apart, which only the indexed copies read
        xyz = torch.randn((3, n + 3), generator=g).cuda().t()
    attr = torch.randint(-2**31, 2**31 - 1, (n + 3,), generator=g).to(torch.int32).cuda()
    t = torch.randn(n + 3, generator=g).cuda()
    frame = torch.randint(0, 99, (n + 3,), generator=g).to(torch.int32).cuda()
    return xyz, attr, t, frame


@pytest.mark.parametrize("form,width", [("rows", 3), ("rows", 4), ("view", 3), ("shifted", 4), ("columns", 3)])
def test_ring_append(form, width):
    cap = 1000
    pipe = gpu.Pipeline(ring_capacity=cap, map_capacity=1 << 10)
    want = [np.zeros((cap, 3), np.float32)] + [np.zeros(cap, d) for d in (np.int32, np.float32, np.int32)]
    head = filled = 0
    for k, n in enumerate((1, 255, 256, 600, 0, 999, 1000, 2300, 3)):  # inside, across the end, more than the ring
        xyz, attr, t, frame = _batch(n, width, form, k)
        pipe.ingest_ring(xyz, attr if k % 2 else attr.view(torch.uint32), t, frame, n)
        keep = min(n, cap)
        at = (head + np.arange(keep)) % cap
        for w, x in zip(want, (xyz[:, :3], attr, t, frame)):
            w[at] = x.cpu().numpy()[n - keep:n]
        head, filled = (head + keep) % cap, min(filled + keep, cap)
        assert (pipe.head, pipe.filled) == (head, filled)
        for w, x in zip(want, (pipe.ring_xyz, pipe.ring_attr, pipe.ring_t, pipe.ring_frame)):
            np.testing.assert_array_equal(w.view(np.uint32), x.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("m,m_ub", [(0, 1), (1, 1), (700, 1000), (1200, 1000), (1000, 1000)])
def test_frame_copy(m, m_ub):
    cap = 1000
    xyz, attr, t, frame = _batch(cap, 4, "rows", m)
    count = torch.tensor([m], dtype=torch.int32, device="cuda")
    fb = _lib.FrameBuf()
    fb.f_xyz, fb.f_attr, fb.f_t, fb.f_frame = (x.data_ptr() for x in (xyz, attr, t, frame))
    out = [torch.full_like(x, 7) for x in (xyz, attr, t, frame)] + [torch.zeros_like(count)]
    _lib.call("lw_frame_copy", ctypes.byref(fb), _lib.ptr(count), m_ub, *(_lib.ptr(x) for x in out), _lib.stream_ptr())
    n = min(m, m_ub)
    for x, y in zip((xyz, attr, t, frame), out):
        assert torch.equal(y[:n], x[:n]) and bool((y[n:] == 7).all())
    assert int(out[4]) == m
