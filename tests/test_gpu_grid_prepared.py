"""Prepared maps that were changed after prepare(), or put together elsewhere: `start` is what counts, and any numeric arrays
of the right shapes serve."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _host(n=3000, seed=2):
    from livox_warp.mapgrid import PriorGrid

    rng = np.random.default_rng(seed)
    xyz = (rng.uniform(0.0, 1.0, (n, 3)) * (2.0, 1.5, 0.8)).astype(np.float32)
    return PriorGrid.prepare({"xyz": xyz, "normal": rng.normal(0.0, 1.0, (n, 3)).astype(np.float32),
                              "planarity": rng.uniform(0.0, 1.0, n).astype(np.float32)})


def _build(host):
    from livox_warp.mapgrid import PriorGrid

    grid = PriorGrid(host)
    grid.build()
    return grid


def _same(a, b):
    return all(torch.equal(x, y) for x, y in ((a.start, b.start), (a.nn, b.nn), (a.df, b.df), (a.xyzp, b.xyzp),
                                              (a.nrm, b.nrm)))


def _keep(host, mask):
    """The map without some of its points, its prefix array brought up to date, what else it holds left as it was."""
    kept = np.concatenate([[0], np.cumsum(mask)]).astype(np.int32)
    return dict(host, xyz=host["xyz"][mask], normal=host["normal"][mask], planarity=host["planarity"][mask],
                start=kept[host["start"]])


@pytest.mark.parametrize("case", ["every other point", "one point", "one point moved to the next cell", "steps cut short",
                                  "steps of another map", "a step beyond the grid"])
def test_the_prefix_array_counts(case):
    host = _host()
    n = len(host["xyz"])
    if case == "every other point":
        host = _keep(host, np.arange(n) % 2 == 0)
    elif case == "one point":
        host = _keep(host, np.arange(n) != 1234)
    elif case == "one point moved to the next cell":  # the array differs in one place
        c = int(host["cells"][500])
        host = dict(host, start=host["start"].copy())
        host["start"][c + 1] -= 1
    elif case == "steps cut short":
        host = dict(host, cells=host["cells"][:-3], first=host["first"][:-3])
    elif case == "steps of another map":
        other = _host(2000, 9)
        host = dict(host, cells=other["cells"], first=other["first"])
    else:
        cells = host["cells"].copy()
        cells[700] = len(host["start"]) + 5
        host = dict(host, cells=cells)
    plain = {k: v for k, v in host.items() if k not in ("cells", "first")}
    a, b = _build(host), _build(plain)
    assert np.array_equal(a.start.cpu().numpy(), host["start"])
    assert _same(a, b)


@pytest.mark.parametrize("case", ["float64", "reversed view", "columns of a wider array", "big-endian", "one planarity",
                                  "int64 steps", "a list"])
def test_other_arrays_of_the_same_values(case):
    host = _host()
    want = _build(host)
    if case == "float64":
        host = dict(host, xyz=host["xyz"].astype(np.float64), planarity=host["planarity"].astype(np.float64))
    elif case == "reversed view":
        host = dict(host, xyz=np.ascontiguousarray(host["xyz"][::-1])[::-1],
                    planarity=np.ascontiguousarray(host["planarity"][::-1])[::-1])
    elif case == "columns of a wider array":
        host = dict(host, xyz=np.concatenate([host["xyz"]] * 2, axis=1)[:, :3])
    elif case == "big-endian":
        host = dict(host, xyz=host["xyz"].astype(">f4"), planarity=host["planarity"].astype(">f4"))
    elif case == "one planarity":
        want = _build(dict(host, planarity=np.full(len(host["xyz"]), 0.75, np.float32)))
        host = dict(host, planarity=0.75)
    elif case == "int64 steps":
        host = dict(host, cells=host["cells"].astype(np.int64), first=host["first"].astype(np.int64))
    else:
        host = dict(host, planarity=host["planarity"].tolist())
    assert _same(_build(host), want)
