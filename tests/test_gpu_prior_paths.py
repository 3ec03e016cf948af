"""The prior-map builder's sums over their whole range: a voxel's sums by bulk reductions and by atomics (whole numbers, so
equal), and normals of clouds with few and with thousands of points per cell against the oracle, bit for bit (whole-number
sums, the same float64 operations on both sides)."""

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("colour,intensity", [(True, True), (False, True), (True, False), (False, False)])
@pytest.mark.parametrize("n", [1, 257, 40_000])
def test_vox_insert_by_reductions_and_by_atomics(n, colour, intensity):
    from livox_warp import _lib, prior_map

    rng = np.random.default_rng(n)
    xyz = rng.uniform(-3.0, 3.0, (n, 3)).astype(np.float32)
    xyz[n // 2:] = xyz[n // 2] + rng.uniform(0.0, 0.02, (n - n // 2, 3)).astype(np.float32)  # many points a voxel
    x = torch.from_numpy(xyz).cuda()
    rgb = torch.from_numpy(rng.uniform(-300.0, 300.0, (n, 3)).astype(np.float32)).cuda() if colour else None
    inten = torch.from_numpy(rng.uniform(-2.0, 2.0, n).astype(np.float32)).cuda() if intensity else None
    out = []
    for aligned in (True, False):
        table = prior_map.VoxelTable(0.05, slots_log2=17, chunk=30_000)
        if not aligned:
            table.acc = torch.empty(table.acc.numel() + 1, dtype=torch.int64, device="cuda")[1:]
            table.buf.acc = table.acc.data_ptr()
            table.clear()
        assert (table.acc.data_ptr() % 16 == 0) == aligned
        table.insert(x, inten, rgb)
        out.append([v.cpu().numpy() for v in table.emit()] + [table.totals()])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    want = oracle.voxel_downsample(xyz, None if inten is None else inten.cpu().numpy(),
                                   None if rgb is None else rgb.cpu().numpy(), 0.05)
    assert np.array_equal(out[0][0], want[0]) and np.array_equal(out[0][3], want[3])


def _cloud(kind, n, rng):
    if kind == "sparse":  # a cell or more per lane
        return rng.uniform(-4.0, 4.0, (n, 3))
    if kind == "surface":
        p = rng.uniform(-1.0, 1.0, (n, 3))
        p[:, 2] = 0.1 * p[:, 0] + rng.normal(0.0, 0.003, n)
        return p
    if kind == "lump":  # every point within the radius of every other, across cell borders
        return rng.normal(0.0, 0.012, (n, 3))
    p = rng.uniform(-1.0, 1.0, (n, 3))  # "mixed": a lump among scattered points, and points that coincide
    p[: n // 3] = rng.normal(0.3, 0.02, (n // 3, 3))
    p[n // 3: n // 2] = p[n // 3]
    return p


@pytest.mark.parametrize("kind", ["sparse", "surface", "lump", "mixed"])
@pytest.mark.parametrize("n", [1, 31, 33, 300, 3000])
def test_normals_bit_exact_over_densities(kind, n):
    from livox_warp import prior_map

    xyz = _cloud(kind, n, np.random.default_rng(n)).astype(np.float32)
    gn, gp = prior_map.normals(xyz, 0.1)
    on, op = oracle.normals(xyz, 0.1)
    assert np.array_equal(gn, on) and np.array_equal(gp, op)
