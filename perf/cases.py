"""The framework's work as its users have it done, as cases that can be timed: one pass through the public entry points
for each path a program takes -- registering a frame, following a recording, keeping a live map, understanding the
visible set, placing scans in a prior map, searching it, building it, training the learned start.

Sizes are those of the repository's own benchmark and tests and the ranges around them: Mid-40-like frames of about
10,000 points (2,000 when thinned or far between, 150,000 from several sensors), registration voxels of 0.1-0.25 m,
integration maps of 0.05-0.1 m, prior maps of 0.5-6M points, 4 to 256 hypotheses of 2,000-20,000 points. Scans are
traced on the GPU into the seeded scenes of livox_warp.synth.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "livox-warp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from livox_warp import gpu, initnet, prior_map, synth  # noqa: E402
from livox_warp.localize import GlobalLocalizer, coarse_positions, score_grid  # noqa: E402
from livox_warp.mapgrid import PriorGrid  # noqa: E402
from livox_warp.odom import Odometry  # noqa: E402
from livox_warp.perception import Perception  # noqa: E402

FRAME_DT = 0.1
GROUND = dict(cell=0.5, thick=0.15, min_sup=3, thresh=0.2, slope_step=0.3)


def listed() -> list[dict]:
    return [
        # a sparse frame (a thinned or 20 kHz sensor) registered from host arrays: all latency, the smallest call
        {"name": "register_sparse", "kind": "register", "points": 2000, "voxel": 0.2, "iters": 10, "host": True},
        # the repository's headline: a 10,000-point Mid-40 frame against a 0.2 m map, at most 10 iterations
        {"name": "register", "kind": "register", "points": 10000, "voxel": 0.2, "iters": 10, "host": True},
        # several sensors' frame already on the device, the odometry's own voxel and iteration limit
        {"name": "register_dense", "kind": "register", "points": 120000, "voxel": 0.15, "iters": 16, "host": False},
        # 2.4 s of a recording through the streaming odometry, every frame inserted and carved, the trajectory read
        {"name": "recording", "kind": "recording", "frames": 24, "points": 10000, "voxel": 0.15, "map_voxel": 0.1},
        # a live view without odometry: a second of batches into the ring and the map, carved, then drawn
        {"name": "live_view", "kind": "live", "batches": 10, "points": 20001, "voxel": 0.1, "every": 2},
        # one perception frame: the map's visible set with normals, ground and clusters, at the viewer's size
        {"name": "perceive", "kind": "perceive", "points": 250000, "voxel": 0.1, "radius": 0.3, "slots_log2": 22,
         "connect": 0.35},
        # the same over a whole scanned floor
        {"name": "perceive_floor", "kind": "perceive", "points": 4000000, "voxel": 0.05, "radius": 0.15,
         "slots_log2": 23, "connect": 0.15},
        # many hypotheses with a scan each, of uneven length, placed in a prior map (the kidnapped robot, a fleet)
        {"name": "locate", "kind": "locate", "hyps": 256, "lo": 2000, "hi": 20000, "size_x": 20.0, "spacing": 0.025},
        # the coarse global search of one gravity candidate: every free position and heading
        {"name": "search", "kind": "search", "points": 1024, "heights": 4, "xy_step": 0.25, "yaws": 180,
         "size_x": 20.0},
        # a scanned cloud with colour and intensity made into a prior map: voxel means, normals, planarity
        {"name": "prior_map", "kind": "prior", "voxels": 1400000, "voxel": 0.02, "radius": 0.08},
        # a prepared map uploaded and its nearest-point grid built (what loading a map costs)
        {"name": "prior_grid", "kind": "grid", "size_x": 20.0, "spacing": 0.03},
        # one optimiser step of the learned start's network
        {"name": "train_step", "kind": "train", "batch": 256, "step": True},
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("register", "register", "recording", "live", "perceive", "perceive", "locate", "search",
                       "prior", "grid", "train"))
    if kind == "register":
        return {"kind": kind, "points": log_int(1000, 120000), "voxel": round(rng.uniform(0.1, 0.25), 3),
                "iters": rng.choice((6, 10, 16)), "host": rng.random() < 0.5}
    if kind == "recording":
        return {"kind": kind, "frames": rng.randint(10, 24), "points": log_int(3000, 10000),
                "voxel": round(rng.uniform(0.12, 0.25), 3), "map_voxel": round(rng.uniform(0.08, 0.15), 3)}
    if kind == "live":
        return {"kind": kind, "batches": rng.randint(3, 10), "points": log_int(1000, 20000),
                "voxel": round(rng.uniform(0.07, 0.2), 3), "every": rng.choice((1, 2, 4))}
    if kind == "perceive":
        voxel = round(rng.uniform(0.06, 0.15), 3)
        return {"kind": kind, "points": log_int(20000, 3000000), "voxel": voxel,
                "radius": round(voxel * rng.uniform(1.5, 3.2), 3), "slots_log2": rng.choice((22, 23)),
                "connect": round(voxel * rng.uniform(1.5, 2.9), 3)}
    if kind == "locate":
        lo = rng.randint(1500, 6000)
        return {"kind": kind, "hyps": log_int(4, 250), "lo": lo, "hi": rng.randint(lo + 500, 20000),
                "size_x": round(rng.uniform(10.0, 20.0), 1), "spacing": round(rng.uniform(0.025, 0.05), 4)}
    if kind == "search":
        return {"kind": kind, "points": rng.randint(300, 1024), "heights": rng.randint(1, 4),
                "xy_step": round(rng.uniform(0.25, 0.5), 3), "yaws": rng.choice((90, 120, 180)),
                "size_x": round(rng.uniform(10.0, 20.0), 1)}
    if kind == "prior":
        voxel = round(rng.uniform(0.02, 0.05), 4)
        return {"kind": kind, "voxels": log_int(30000, 1200000), "voxel": voxel,
                "radius": round(voxel * rng.uniform(2.5, 4.0), 4)}
    if kind == "grid":
        return {"kind": kind, "size_x": round(rng.uniform(8.0, 20.0), 1), "spacing": round(rng.uniform(0.03, 0.06), 4)}
    return {"kind": kind, "batch": log_int(1, 250), "step": rng.random() < 0.6}


def prepare(case: dict, seed: int):
    return _PREPARE[case["kind"]](case, np.random.default_rng(seed), int(seed))


def run(state):
    return _RUN[state["kind"]](state)


def exact(case: dict, seed: int):
    make = _EXACT.get(case["kind"])
    return None if make is None else make(case, np.random.default_rng(seed), int(seed))


def work(case: dict) -> dict:
    return _WORK[case["kind"]](case)


# ---- scenes and scans ----------------------------------------------------------------------------------------------


def _cast(scene, o: torch.Tensor, d: torch.Tensor) -> torch.Tensor:
    """Distance along unit rays d ((n, 3) float64 CUDA, world frame) from o ((3,) or (n, 3)) to the scene's first
    surface: the room from inside, the solid boxes from outside."""
    dev = d.device
    room = torch.from_numpy(np.stack([scene.room_lo, scene.room_hi])).to(dev)
    boxes = torch.from_numpy(np.asarray(scene.boxes, np.float64)).to(dev)
    o = o.expand(len(d), 3)
    out = torch.empty(len(d), dtype=torch.float64, device=dev)
    chunk = max(1024, 4_000_000 // max(len(boxes), 1))
    for a in range(0, len(d), chunk):
        oo, dd = o[a:a + chunk], d[a:a + chunk]
        inv = 1.0 / torch.where(dd.abs() < 1e-12, torch.full_like(dd, 1e-12), dd)
        best = torch.where(dd > 0, (room[1] - oo) * inv, (room[0] - oo) * inv).min(dim=1).values
        t1 = (boxes[None, :, :3] - oo[:, None]) * inv[:, None]
        t2 = (boxes[None, :, 3:] - oo[:, None]) * inv[:, None]
        near = torch.minimum(t1, t2).max(dim=2).values
        far = torch.maximum(t1, t2).min(dim=2).values
        hit = torch.where((near <= far) & (near > 1e-6), near, torch.full_like(near, math.inf))
        out[a:a + chunk] = torch.minimum(best, hit.min(dim=1).values)
    return out


def _scan(scene, T: np.ndarray, d: np.ndarray, rng, noise: float, sizes=None) -> torch.Tensor:
    """Sensor-frame float32 points of rays d ((n, 3), sensor frame), with range noise, from one pose T (4, 4), a pose
    per ray (n, 4, 4) or, with `sizes`, a pose per run of sizes[k] rays."""
    d = torch.from_numpy(d).cuda()
    T = torch.from_numpy(np.ascontiguousarray(T)).cuda()
    if sizes is not None:
        T = torch.repeat_interleave(T, torch.from_numpy(sizes).cuda(), dim=0)
    dw = (T[..., :3, :3] @ d[..., None])[..., 0]
    r = _cast(scene, T[..., :3, 3], dw) + torch.from_numpy(rng.normal(0.0, noise, len(d))).cuda()
    return (d * r[:, None]).float()


def _sphere(n: int, rng, elev=(-45.0, 60.0)) -> np.ndarray:
    az, el = rng.uniform(0.0, 2.0 * math.pi, n), np.radians(rng.uniform(*elev, n))
    return np.stack([np.cos(el) * np.cos(az), np.cos(el) * np.sin(az), np.sin(el)], axis=1)


def _attr(n: int, rng) -> np.ndarray:
    return rng.integers(0, 256, n).astype(np.uint32)  # reflectivity; noise tag 0, first return


def _room_pose() -> np.ndarray:
    """A corner of the box room, looking across it and slightly down."""
    return synth.look_at([0.8, 0.8, 1.6], [7.0, 5.0, 1.0])


def _office(size_x: float, seed: int):
    """A stretch of the office: its room grid and box count scaled to the floor's size."""
    return synth.office(seed, size=(size_x, 0.75 * size_x, 3.0), rooms=(max(2, round(size_x / 10.0)), 1),
                        n_boxes=int(size_x))


# ---- one frame against a registration map --------------------------------------------------------------------------


def _register_frame(case, rng, seed):
    """The map's frames (the sensor at rest) and one frame taken while it moves, with its start and body twist."""
    n, scene, T0 = case["points"], synth.box_room(seed % 1000), _room_pose()
    t = FRAME_DT * np.arange(10 * n) / n
    base = _scan(scene, T0, synth.rosette_dirs(t), rng, 0.02)
    t0 = 1.0
    tm = t0 + FRAME_DT * np.arange(n) / n
    mover = synth.ConstantVelocity(T0, t0, 0.5, math.radians(20.0))
    xyz = _scan(scene, mover.poses(tm), synth.rosette_dirs(tm), rng, 0.02)
    # the body motion per frame as a smoothed odometry knows it, a few per cent off
    twist = np.array([0.05, 0.0, 0.0, 0.0, 0.0, math.radians(2.0)]) * rng.uniform(0.95, 1.05, 6)
    return T0, base, t.astype(np.float32), xyz, tm.astype(np.float32), t0 + 0.5 * FRAME_DT, twist.astype(np.float32)


def _prepare_register(case, rng, seed):
    T0, base, tb, xyz, t, t_mid, twist = _register_frame(case, rng, seed)
    n = case["points"]
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << 16)
    odom = Odometry(pipe, reg_slots=1 << 21, frame_cap=1 << 18)
    odom.reg_voxel, odom.max_iter = case["voxel"], case["iters"]
    odom.reset(T0)
    attr = _attr(10 * n, rng).view(np.int32)
    for k in range(10):
        x4 = torch.cat([base[k * n:(k + 1) * n], torch.from_numpy(tb[k * n:(k + 1) * n, None]).cuda()], 1)
        odom.insert_frame(x4.contiguous(), torch.from_numpy(attr[k * n:(k + 1) * n].copy()).cuda(), T0)
    at = _attr(n, rng)
    s = {"kind": "register", "odom": odom, "n": n, "t_mid": t_mid, "twist": twist, "T": T0, "host": case["host"]}
    if case["host"]:
        s.update(xyz=xyz.cpu().numpy(), attr=at, t=t)
    else:
        s.update(xyz=torch.cat([xyz, torch.from_numpy(t[:, None]).cuda()], 1).contiguous(),
                 attr=torch.from_numpy(at.view(np.int32)).cuda(), t=None)
    return s


def _run_register(s):
    odom = s["odom"]
    T, ok, st = odom.register_frame(s["xyz"], s["attr"], s["t"], s["t_mid"], s["twist"], s["T"])
    # the pose in float32, as the pose table and the maps take it, and the deskewed frame (x, y, z, t)
    return {"T": T.astype(np.float32), "ok": ok, "iters": st["iters"], "ds": st["ds"], "corr": st["corr"],
            "frame": odom.f_xyz[:s["n"]]}


def _exact_register(case, rng, seed):
    """The deskewed frame in float64. The pose is where an iteration stops: it has no closed value to hold it to."""
    *_, xyz, t, t_mid, twist = _register_frame(case, rng, seed)
    x, tw = xyz.double().cpu().numpy(), twist.astype(np.float64)
    s = (t.astype(np.float64) - t_mid) / FRAME_DT
    a = np.linalg.norm(tw[3:])
    k = tw[3:] / a
    c, sn = np.cos(a * s)[:, None], np.sin(a * s)[:, None]
    rot = x * c + np.cross(k, x) * sn + k * (x @ k)[:, None] * (1.0 - c)
    return {"T": None, "ok": None, "iters": None, "ds": None, "corr": None,
            "frame": np.concatenate([rot + tw[:3] * s[:, None], t[:, None].astype(np.float64)], 1)}


def _work_register(case):
    # the frame read and written once, the thinned points and the map records they meet read in every iteration
    n = case["points"]
    ds = min(n, 2500.0 * (0.2 / case["voxel"]) ** 2)
    return {"bytes": 36.0 * n + case["iters"] * ds * (16 + 80), "flops": 60.0 * n + case["iters"] * ds * 400.0}


# ---- a recording through the streaming odometry ----------------------------------------------------------------------


def _prepare_recording(case, rng, seed):
    n, m, T0 = case["points"], case["frames"], _room_pose()
    scene = synth.box_room(seed % 1000)
    t = FRAME_DT * np.arange(m * n) / n
    mover = synth.ConstantVelocity(T0, 0.8, 0.5, math.radians(20.0))
    xyz = _scan(scene, mover.poses(t), synth.rosette_dirs(t), rng, 0.02).cpu().numpy()
    attr, t32 = _attr(m * n, rng), t.astype(np.float32)
    frames = [(xyz[k:k + n].copy(), attr[k:k + n].copy(), t32[k:k + n].copy()) for k in range(0, m * n, n)]
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << 22)
    odom = Odometry(pipe)
    odom.reg_voxel = case["voxel"]
    odom.integrate(gpu.make_view(voxel=case["map_voxel"], map_cap=pipe.map_cap), case["map_voxel"], overlap=True)
    return {"kind": "recording", "pipe": pipe, "odom": odom, "T0": T0, "frames": frames}


def _run_recording(s):
    pipe, odom = s["pipe"], s["odom"]
    odom.reset(s["T0"])
    pipe.clear_map()
    for x, a, t in s["frames"]:
        sx, sa, st, _ = pipe.stage(x, a, t, len(t), 1.0 / FRAME_DT)
        odom.push(sx, sa, st, len(t), float(t[0]), float(t[-1]))
    odom.flush()
    return np.stack([T for _, _, T in odom.traj]).astype(np.float32)


def _work_recording(case):
    n = case["points"]
    # per frame: registered, inserted (read, one voxel line each), and some 60 voxels' keys along each ray
    return {"bytes": case["frames"] * (n * (36 + 24 + 64) + n * 60 * 8.0), "flops": case["frames"] * n * 60 * 12.0}


# ---- a live view without odometry ------------------------------------------------------------------------------------


def _live_batches(case, rng, seed):
    n, m, T0 = case["points"], case["batches"], _room_pose()
    scene = synth.box_room(seed % 1000)
    walker = np.array([[2.0, 2.0, 0.0, 2.4, 2.4, 1.8]])
    still = scene.boxes
    out = []
    for k in range(m):
        t = FRAME_DT * (k + np.arange(n) / n)
        scene.boxes = np.concatenate([still, walker + np.array([0.12 * k, 0.08 * k, 0.0] * 2)])
        out.append((_scan(scene, T0, synth.rosette_dirs(t), rng, 0.02).cpu().numpy(), _attr(n, rng),
                    t.astype(np.float32)))
    return T0, out


def _prepare_live(case, rng, seed):
    T0, batches = _live_batches(case, rng, seed)
    pipe = gpu.Pipeline(ring_capacity=1 << 20, map_capacity=1 << 20)
    pipe.set_pose(0, T0)
    now = FRAME_DT * case["batches"]
    view = gpu.make_view(now=now, voxel=case["voxel"], map_cap=pipe.map_cap, carve_on=1, dyn_on=1, dyn_settle=0.5 * now)
    return {"kind": "live", "pipe": pipe, "view": view, "batches": batches, "voxel": case["voxel"],
            "every": case["every"]}


def _run_live(s):
    pipe, view = s["pipe"], s["view"]
    pipe.clear_live()
    pipe.clear_map()
    for x, a, t in s["batches"]:
        n = len(t)
        sx, sa, st, sf = pipe.stage(x, a, t, n)
        pipe.ingest_ring(sx, sa, st, sf, n)
        pipe.map_insert(sx, sa, st, sf, n, view, s["voxel"])
        pipe.carve(sx, sa, sf, n, s["voxel"], every=s["every"])
    n = pipe.build(view, map_on=False)
    return {"xyz": pipe.c_xyz[:n], "attr": pipe.c_attr[:n], "t": pipe.c_t[:n], "moving": pipe.c_dyn[:n],
            "voxels": pipe.map_stats}


def _exact_live(case, rng, seed):
    """Every point in range is drawn, in ring order, at its pose."""
    T0, batches = _live_batches(case, rng, seed)
    x = np.concatenate([b[0] for b in batches]).astype(np.float64)
    return {"xyz": x @ T0[:3, :3].T + T0[:3, 3], "attr": None,
            "t": np.concatenate([b[2] for b in batches]).astype(np.float64), "moving": None, "voxels": None}


def _work_live(case):
    n = case["points"] * case["batches"]
    return {"bytes": n * (20.0 + 24 + 64 + 44) + n / case["every"] * 60 * 8.0, "flops": n / case["every"] * 60 * 12.0}


# ---- the map's visible set: normals, ground, clusters ----------------------------------------------------------------


def _floor_points(case, rng, seed):
    """A scanned floor in world coordinates: rays from a few stations of the office."""
    scene = _office(16.0, seed % 1000)
    stations = synth.free_poses(scene, 4, seed, z=1.4)
    n = case["points"]
    parts = []
    for k in range(4):
        m = n // 4 + (k < n % 4)
        local = _scan(scene, stations[k], _sphere(m, rng), rng, 0.01)
        T = torch.from_numpy(stations[k]).cuda()
        parts.append((local.double() @ T[:3, :3].T + T[:3, 3]).float())
    return torch.cat(parts)


def _voxel_order(xyz: torch.Tensor, voxel: float, slots_log2: int):
    """(each voxel's first point, the voxel of every point, the voxels in the order of their home slots)."""
    ijk = torch.floor(xyz * np.float32(1.0 / voxel)).to(torch.int64).cpu().numpy()
    key = gpu.voxel_key_ijk(ijk[:, 0], ijk[:, 1], ijk[:, 2])
    uniq, first, inv = np.unique(key, return_index=True, return_inverse=True)
    h = uniq * np.int64(gpu.HASH_MULTIPLIER)
    home = (h ^ (h >> np.int64(29))) & np.int64((1 << slots_log2) - 1)
    return first, inv.reshape(-1), np.argsort(home, kind="stable"), home


def _prepare_perceive(case, rng, seed):
    """A map holding the floor. Voxels are opened by their first points, sixteenth by sixteenth of the table, so that
    voxels with the same home slot always come in the same order; the other points follow in one batch."""
    xyz = _floor_points(case, rng, seed)
    n = len(xyz)
    first, _, order, _ = _voxel_order(xyz, case["voxel"], case["slots_log2"])
    pipe = gpu.Pipeline(ring_capacity=1 << 16, map_capacity=1 << case["slots_log2"])
    view = gpu.make_view(now=1.0, voxel=case["voxel"], map_cap=pipe.map_cap)
    attr = torch.from_numpy(_attr(n, rng).view(np.int32)).cuda()
    t = torch.linspace(0.0, 1.0, n, device="cuda")
    later = np.ones(n, bool)
    later[first] = False
    for idx in [first[order[k::16]] for k in range(16)] + [np.flatnonzero(later)]:
        i = torch.from_numpy(idx).cuda()
        pipe.map_insert(xyz[i].contiguous(), attr[i].contiguous(), t[i].contiguous(),
                        torch.zeros(len(i), dtype=torch.int32, device="cuda"), len(i), view, case["voxel"])
    perc = Perception(pipe)
    return {"kind": "perceive", "pipe": pipe, "perc": perc, "view": view, "radius": case["radius"],
            "voxel": case["voxel"], "connect": case["connect"], "rows": min(n, pipe.work_cap)}


def _run_perceive(s):
    pipe, perc = s["pipe"], s["perc"]
    pipe.build(s["view"], neighbors="normals", radius=s["radius"], sensor=(8.0, 6.0, 1.4))
    perc.ground(use_normals=True, **GROUND)
    found = perc.cluster(voxel=s["voxel"], connect=s["connect"])
    table = np.zeros((gpu.MAX_CLUSTERS, 10), np.float32)
    for j, c in enumerate(found):
        table[j] = (c["cnt"], *c["cen"], *c["lo"], *c["hi"])
    n = s["rows"]  # the visible set's buffers, as far as these points can fill them
    return {"xyz": pipe.c_xyz[:n], "attr": pipe.c_attr[:n], "t": pipe.c_t[:n], "moving": pipe.c_dyn[:n],
            "neighbours": pipe.nbr[:n], "normal": pipe.nrm[:n], "curvature": pipe.curv[:n], "ground": pipe.gnd[:n],
            "height": pipe.hag[:n], "cluster": pipe.cid[:n], "clusters": table, "visible": pipe.count}


def _exact_perceive(case, rng, seed):
    """The visible points in the table's order, as float64 means of their voxels' points, and the last hit times.
    The labels and what follows from them are decisions on those points."""
    xyz = _floor_points(case, rng, seed)
    n = len(xyz)
    first, inv, order, home = _voxel_order(xyz, case["voxel"], case["slots_log2"])
    cap = 1 << case["slots_log2"]
    taken, slot = np.zeros(cap, bool), np.full(len(first), -1, np.int64)
    for k in range(16):  # linear probing, a sixteenth at a time
        want = order[k::16]
        for p in range(64):
            s = (home[want] + p) & (cap - 1)
            free = ~taken[s]
            slot[want[free]] = s[free]
            taken[s[free]] = True
            want = want[~free]
    cnt = np.bincount(inv, minlength=len(first))
    first_hits = np.minimum(cnt, gpu.MAP_COUNT_CAP)
    x = xyz.double().cpu().numpy()
    if (cnt > gpu.MAP_COUNT_CAP).any():
        return None  # only the first hits of such a voxel are summed
    mean = np.stack([np.bincount(inv, x[:, c], len(first)) for c in range(3)], 1) / first_hits[:, None]
    last = np.zeros(len(first))
    np.maximum.at(last, inv, torch.linspace(0.0, 1.0, n, device="cuda").double().cpu().numpy())
    rows = np.argsort(slot)
    out_xyz, out_t = np.zeros((min(n, cap), 3)), np.zeros(min(n, cap))
    out_xyz[:len(rows)], out_t[:len(rows)] = mean[rows], last[rows]
    return {"xyz": out_xyz, "attr": None, "t": out_t, "moving": None, "neighbours": None, "normal": None,
            "curvature": None, "ground": None, "height": None, "cluster": None, "clusters": None, "visible": None}


def _work_perceive(case):
    # the table's keys once, then per visible voxel its line, its neighbourhood's voxels and the outputs
    m = min(case["points"], 600.0 / case["voxel"] ** 2)
    return {"bytes": 8.0 * (1 << case["slots_log2"]) + m * (64 + 40 + 20 + 27 * 8 + 24), "flops": m * 2000.0}


# ---- the prior map: grid, search, batched registration ------------------------------------------------------------------


def _site(size_x: float, spacing: float, seed: int):
    scene = _office(size_x, seed % 1000)
    xyz, nrm = synth.sample_surfaces(scene, spacing, seed, jitter=0.002)
    return scene, {"xyz": xyz, "normal": nrm}


def _prepare_grid(case, rng, seed):
    _, host = _site(case["size_x"], case["spacing"], seed)
    return {"kind": "grid", "grid": PriorGrid(host)}


def _run_grid(s):
    s["grid"].build()
    return {"nearest": s["grid"].nn, "distance": s["grid"].df}


def _grid_cells(size_x):
    return (size_x + 1.2) * (0.75 * size_x + 1.2) * (3.0 + 1.2) / 0.05 ** 3


def _site_points(size_x, spacing):
    return (2.0 * 0.75 * size_x ** 2 + 3.5 * size_x * 3.0 + 5.0 * size_x + 4.0 * size_x) / spacing ** 2


def _work_grid(case):
    cells = _grid_cells(case["size_x"])
    return {"bytes": 28.0 * _site_points(case["size_x"], case["spacing"]) + cells * (4 + 4 + 1),
            "flops": cells * 20.0}


def _prepare_locate(case, rng, seed):
    scene, host = _site(case["size_x"], case["spacing"], seed)
    grid = PriorGrid(host)
    grid.build()
    k = case["hyps"]
    sizes = rng.integers(case["lo"], case["hi"] + 1, k)
    true = synth.free_poses(scene, k, seed, z=1.2)
    hi = np.cumsum(sizes)
    lo = hi - sizes
    d = _sphere(int(hi[-1]), rng, (-7.0, 52.0))
    pts = _scan(scene, true, d, rng, 0.01, sizes)
    pts4 = torch.zeros((len(pts), 4), dtype=torch.float32).pin_memory()
    pts4[:, :3].copy_(pts)
    loc = GlobalLocalizer(grid, hyp_cap=k, pts_cap=len(pts))
    # the launch shape an installation has settled on, so that a first batch is not spent on trying shapes
    return {"kind": "locate", "loc": loc, "pts": pts4, "lo": lo, "hi": hi, "tile": 32, "ctas": 5,
            "T": synth.perturb(true, seed + 1, 0.25, 2.5, 0.5)}


def _run_locate(s):
    r = s["loc"].register_packed(s["pts"], s["lo"], s["hi"], s["T"], tile=s["tile"], blocks_per_sm=s["ctas"])
    # the poses in float32, as a scan's points are posed; the fit is counts over points
    return {"T": r.T.astype(np.float32), "fit": r.fit.astype(np.float32), "count": r.count, "iters": r.iters}


def _work_locate(case):
    pts = case["hyps"] * 0.5 * (case["lo"] + case["hi"])
    m = _site_points(case["size_x"], case["spacing"])
    return {"bytes": 16.0 * pts + 28.0 * m + 9.0 * _grid_cells(case["size_x"]), "flops": 30 * pts * 250.0}


def _search_inputs(case, rng, seed):
    scene, host = _site(case["size_x"], 0.04, seed)
    T = synth.free_poses(scene, 1, seed, z=1.2)[0]
    pts = _scan(scene, T, _sphere(case["points"], rng, (-7.0, 52.0)), rng, 0.01)
    prep = PriorGrid.prepare(host)
    heights = [1.2 + 0.08 * k for k in range(case["heights"])]
    pos, _, ny = coarse_positions(prep["lo"], prep["hi"], heights, case["xy_step"])
    return prep, pts, pos, ny


def _prepare_search(case, rng, seed):
    prep, pts, pos, ny = _search_inputs(case, rng, seed)
    grid = PriorGrid(prep)
    grid.build()
    return {"kind": "search", "grid": grid, "pts": pts, "pos": torch.from_numpy(pos).cuda(), "ny": ny,
            "yaws": case["yaws"], "out": torch.empty(len(pos) * case["yaws"], dtype=torch.float32, device="cuda")}


def _run_search(s):
    score_grid(s["grid"], s["pts"], s["pos"], s["yaws"], 0.0, 2.0 * math.pi / s["yaws"], 25.0, 10.0, s["out"],
               pos_stride=s["ny"])
    return s["out"]


def _work_search(case):
    n = (case["size_x"] / case["xy_step"] + 1) * (0.75 * case["size_x"] / case["xy_step"] + 1) * case["heights"]
    h = n * case["yaws"]
    # each hypothesis rotates every point once (6), adds its position (3), finds its cell (6) and adds (2)
    return {"bytes": _grid_cells(case["size_x"]) + 4.0 * h, "flops": h * case["points"] * 17.0}


def _cloud(case, rng, seed):
    """A cloud of a building's surfaces, about 2.5 points to a voxel, in runs of neighbouring points as a scanner gives
    them, cut off where its last voxel opens (so that every seed has the same number of voxels)."""
    voxels, voxel = case["voxels"], case["voxel"]
    size = max(8.0, math.sqrt(0.75 * voxels) * voxel)
    xyz, _ = synth.sample_surfaces(_office(size, seed % 1000), voxel / 1.6, seed, jitter=0.002)
    runs = rng.permutation(len(xyz) // 512)
    xyz = xyz[:len(runs) * 512].reshape(-1, 512, 3)[runs].reshape(-1, 3)
    _, first, _ = _voxels_of(torch.from_numpy(xyz).cuda(), voxel)
    n = int(torch.sort(first).values[voxels]) if len(first) > voxels else len(xyz)
    inten, rgb = rng.uniform(0.0, 1.0, n).astype(np.float32), rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    return tuple(torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (xyz[:n], inten, rgb))


def _voxels_of(xyz: torch.Tensor, voxel: float):
    """(the voxel of every point, each voxel's first point, each voxel's count), voxels in the order of their keys."""
    ijk = torch.floor(xyz * np.float32(1.0 / float(np.float32(voxel)))).to(torch.int64) + (1 << 20)
    _, inv, cnt = torch.unique(ijk[:, 0] | ijk[:, 1] << 21 | ijk[:, 2] << 42, return_inverse=True, return_counts=True)
    at = torch.arange(len(xyz), device=xyz.device)
    first = torch.full_like(cnt, len(xyz)).scatter_reduce_(0, inv, at, "amin")
    return inv, first, cnt


def _prepare_prior(case, rng, seed):
    xyz, inten, rgb = _cloud(case, rng, seed)
    # tables sized once for what the building may hold
    table = prior_map.VoxelTable(case["voxel"], max(16, (4 * case["voxels"] - 1).bit_length()), chunk=len(xyz))
    return {"kind": "prior", "xyz": xyz, "inten": inten, "rgb": rgb, "table": table, "radius": case["radius"],
            "bufs": prior_map.NormalBuffers(case["voxels"])}


def _run_prior(s):
    table = s["table"]
    table.clear()
    table.insert(s["xyz"], s["inten"], s["rgb"])
    xyz, rgb, inten, cnt = table.emit()
    nrm, planar = prior_map.normals_device(xyz, s["radius"], bufs=s["bufs"])
    return {"xyz": xyz, "rgb": rgb, "intensity": inten, "count": cnt, "normal": nrm, "planarity": planar}


def _exact_prior(case, rng, seed):
    """Float64 means of each voxel's points, voxels in the order of their first point. The normals' signs and the
    planarity belong to the float32 means they are taken from."""
    xyz, inten, rgb = _cloud(case, rng, seed)
    inv, first, cnt = _voxels_of(xyz, case["voxel"])
    order = torch.argsort(first)

    def mean(v):
        s = torch.zeros((len(first), v.shape[1]), dtype=torch.float64, device="cuda").index_add_(0, inv, v.double())
        return (s / cnt[:, None])[order]

    return {"xyz": mean(xyz), "rgb": mean(rgb), "intensity": mean(inten[:, None])[:, 0], "count": None,
            "normal": None, "planarity": None}


def _work_prior(case):
    m = case["voxels"]
    near = math.pi * (case["radius"] / case["voxel"]) ** 2
    return {"bytes": 28.0 * 2.5 * m + m * (32 + 12 + 16), "flops": m * near * 20.0}


# ---- the learned start -----------------------------------------------------------------------------------------------


def _pairs(case, rng, seed):
    """Frame and map point sets around the sensor, as the odometry cuts them, and the steps to learn."""
    n, P = case["batch"], initnet.P
    scene = synth.box_room(seed % 1000)
    d = synth.rosette_dirs(rng.uniform(0.0, 1.0, 2 * n * P))
    sets = torch.zeros((2 * n, P, 4), dtype=torch.float32, device="cuda")
    sets[..., :3] = _scan(scene, _room_pose(), d, rng, 0.02).view(2 * n, P, 3)
    target = torch.from_numpy(rng.normal(0.0, 1.0, (n, 6)) * np.asarray(initnet.OUT_SCALE)).float().cuda()
    return sets, target


_LAYERS = (("W1", (64, 3)), ("B1", (64,)), ("W2", (128, 64)), ("B2", (128,)), ("W3", (256, 128)), ("B3", (256,)),
           ("WH1", (128, 512)), ("BH1", (128,)), ("WH2", (6, 128)), ("BH2", (6,)))


def _weights(seed: int) -> np.ndarray:
    """A network part-way through its training: weights of the usual spread, small biases."""
    rng = np.random.default_rng(seed + 77)
    w = np.zeros(initnet.NPARAM, np.float32)
    for name, shape in _LAYERS:
        size = int(np.prod(shape))
        spread = math.sqrt(2.0 / shape[1]) if len(shape) == 2 else 0.05
        w[initnet.OFF[name]:initnet.OFF[name] + size] = rng.normal(0.0, spread, size)
    return w


def _prepare_train(case, rng, seed):
    sets, target = _pairs(case, rng, seed)
    net = initnet.InitNet(seed=0, batch_cap=case["batch"])
    net.load_state_dict({"master": _weights(seed), "out_scale": np.asarray(initnet.OUT_SCALE, np.float32),
                         "in_scale": 0.125})
    return {"kind": "train", "net": net, "sets": sets, "target": target, "n": case["batch"], "step": case["step"]}


def _run_train(s):
    net, n = s["net"], s["n"]
    fwd = net.forward(s["sets"], n)
    if not s["step"]:
        return {"step": fwd["step"]}
    loss = net.backward(s["sets"], n, fwd, s["target"])
    net.adam(1e-4)
    return {"step": fwd["step"], "loss": loss, "grad": net.grad, "weights": net.master}


def _exact_train(case, rng, seed):
    """The proposed steps in float64, from the bf16 weights. The gradients follow the point that wins each channel."""
    sets, _ = _pairs(case, rng, seed)
    w = torch.from_numpy(_weights(seed)).bfloat16().double().cuda()
    p = {name: w[initnet.OFF[name]:initnet.OFF[name] + int(np.prod(shape))].view(shape) for name, shape in _LAYERS}
    x = sets[..., :3].double() * 0.125
    pooled = []
    for a in range(0, len(x), 32):
        h = torch.relu(x[a:a + 32] @ p["W1"].T + p["B1"])
        h = torch.relu(h @ p["W2"].T + p["B2"])
        pooled.append(torch.relu(h @ p["W3"].T + p["B3"]).amax(dim=1))
    code = torch.cat(pooled).view(case["batch"], 512)
    out = torch.relu(code @ p["WH1"].T + p["BH1"]) @ p["WH2"].T + p["BH2"]
    step = out * torch.tensor(initnet.OUT_SCALE, dtype=torch.float64, device="cuda")
    return {"step": step, "loss": None, "grad": None, "weights": None} if case["step"] else {"step": step}


def _work_train(case):
    P, n = initnet.P, case["batch"]
    fwd = 2.0 * n * 2 * P * (3 * 64 + 64 * 128 + 128 * 256) + 2.0 * n * (512 * 128 + 128 * 6)
    # backward through the max: one point per channel of each set
    back = 4.0 * n * 2 * 256 * (3 * 64 + 64 * 128 + 128) if case["step"] else 0.0
    return {"bytes": 2.0 * n * P * 16 + 2.0 * initnet.NPARAM + (20.0 * initnet.NPARAM if case["step"] else 0.0),
            "flops": fwd + back}


_PREPARE = {"register": _prepare_register, "recording": _prepare_recording, "live": _prepare_live,
            "perceive": _prepare_perceive, "grid": _prepare_grid, "locate": _prepare_locate,
            "search": _prepare_search, "prior": _prepare_prior, "train": _prepare_train}
_RUN = {"register": _run_register, "recording": _run_recording, "live": _run_live, "perceive": _run_perceive,
        "grid": _run_grid, "locate": _run_locate, "search": _run_search, "prior": _run_prior, "train": _run_train}
_EXACT = {"register": _exact_register, "live": _exact_live, "perceive": _exact_perceive, "prior": _exact_prior,
          "train": _exact_train}
_WORK = {"register": _work_register, "recording": _work_recording, "live": _work_live, "perceive": _work_perceive,
         "grid": _work_grid, "locate": _work_locate, "search": _work_search, "prior": _work_prior,
         "train": _work_train}
