"""Normals of clouds around the line between few points a cell (a lane per point looks its cells up) and many (a warp looks
its few cells up together), 2.5 points a cell, against the oracle, bit for bit."""

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

RADIUS = 0.1
CELL = RADIUS * 1.00390625


@pytest.mark.parametrize("over", [-1, 0, 1])
@pytest.mark.parametrize("cells", [2, 14, 128, 2000])
def test_around_two_and_a_half_points_a_cell(cells, over):
    from livox_warp import prior_map

    rng = np.random.default_rng(cells + over)
    side = int(np.ceil(np.sqrt(cells)))
    ij = np.stack(np.divmod(np.arange(cells), side) + (np.zeros(cells, int),), -1)
    pick = np.concatenate([np.arange(cells)] * 2 + [np.arange(cells // 2)])  # five points to two cells
    pick = pick[:-1] if over < 0 else np.concatenate([pick, np.zeros(over, int)])
    assert len(pick) * 2 == 5 * cells + 2 * over
    xyz = (ij[pick] + 0.5 + rng.uniform(-0.45, 0.45, (len(pick), 3)) * (1, 1, 0.2)) * CELL
    xyz = rng.permutation(xyz).astype(np.float32)
    gn, gp = prior_map.normals(xyz, RADIUS)
    on, op = oracle.normals(xyz, RADIUS)
    assert np.array_equal(gn, on) and np.array_equal(gp, op)
    assert len(xyz) < 30 or (gn != 0).any()
