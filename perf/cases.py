"""Cases that time the frame path through its public entry points.

Each case is one thing a user has the framework do: draw a frame of one view
(`View.frame`, `Engine.frame`), draw one sample of many views (`Batch`), build
lot tables, query rays, serve frames to host memory, shade with the material
surrogate.  `listed()` names the cases, `draw()` gives more of the same ranges,
`prepare()` builds what the program holds before the call, `run()` is one pass.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import stratum_hyperdetail_b200 as sb
from stratum_hyperdetail_b200 import rays as sr
from stratum_hyperdetail_b200.batch import Batch
from stratum_hyperdetail_b200.engine import Engine
from stratum_hyperdetail_b200.server import Pose, Server
from stratum_hyperdetail_b200.views import View

WORLD_SEED = 0x5EED
TUNE = (64, 1, 1)  # block size 64, one tile per claim, Morton order: the server's default

# Camera poses by what they look at: (lot address x, z), position in that lot
# (metres), yaw, pitch.  Streets run along the lot edges (x or z = +-18 m), a
# canal along every lot column with x % 64 == 28.
POSES = {
    "street": ((0, 0), (17.0, 1.7, 0.0), 0.0, 0.0),
    "rooftop": ((0, 0), (17.0, 40.0, 0.0), math.pi / 2, 0.0),
    "aerial": ((0, 0), (0.0, 300.0, 0.0), 0.6, -math.pi / 6),
    "canal": ((28, 1), (0.0, 0.5, 0.0), 0.0, 0.0),
    "park": ((1, 8), (0.0, 2.0, -16.0), 0.0, 0.0),
    "avenue": ((0, 0), (17.99, 12.0, 0.0), 0.0, -2.0 * math.pi / 180),
}

# FP32 operations of the reference algorithm per primary ray (trace, shade and
# resolve; mean of the six poses at 1600x900), per feature the grammar emits in
# bounds mode, and features per lot.
OPS_PER_RAY = 12491.0
OPS_PER_FEATURE = 30.0
FEATURES_PER_LOT = 1859.0
PIXEL_BYTES = 16 + 16 + 16 + 2 * 16 + 4  # Hit, Surface, Linear, History in and out, Pixels
TABLE_BYTES = sb.WORLD_LOTS * (16 * 4 + 4 * 4)  # descriptors and tags of one lot table


def listed():
    return [
        # an interactive preview: the smallest frame a viewer redraws, where launches and latency count
        {"name": "preview_320x180", "kind": "frame", "pose": "street", "width": 320, "height": 180},
        # the plain single-view frame at the headline size, stationary camera accumulating samples
        {"name": "frame_1600x900", "kind": "frame", "pose": "street", "width": 1600, "height": 900},
        # a large still from above, where neighbouring rays diverge most
        {"name": "still_3840x2160", "kind": "frame", "pose": "aerial", "width": 3840, "height": 2160},
        # the engine's loop with a moving camera on a window whose size is no multiple of a tile
        {"name": "engine_walk_1283x721", "kind": "engine", "width": 1283, "height": 721},
        # the headline workload: six views a launch, the captured graph replayed
        {"name": "batch_6x1600x900", "kind": "batch", "views": 6, "width": 1600, "mixed": False, "graph": True},
        # many users' views in one launch: sizes, worlds, heights and directions all different
        {"name": "batch_12_mixed", "kind": "batch", "views": 12, "width": 1920, "mixed": True, "graph": False},
        # streaming: a camera that enters a new column of lots with every frame
        {"name": "flight_1024x576", "kind": "flight", "width": 1024, "height": 576},
        # new worlds: every lot of eight tables described and its hierarchy built
        {"name": "build_8_tables", "kind": "build", "views": 8, "columns": 128},
        # visibility queries of arbitrary rays through the hierarchy
        {"name": "rays_65536", "kind": "rays", "rays": 65536, "exhaustive": False},
        # the same without the hierarchy, as its check runs them
        {"name": "rays_exhaustive_8192", "kind": "rays", "rays": 8192, "exhaustive": True},
        # eight sessions of a render server, one request each, frames in host memory
        {"name": "serve_8", "kind": "serve", "sessions": 8, "width": 1600},
        # one training step of the material surrogate on a traced frame, then its shading
        {"name": "surrogate_1600x900", "kind": "surrogate", "pose": "street", "width": 1600, "height": 900},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "engine", "batch", "batch", "flight", "build", "rays", "serve", "surrogate"])
    pose = rng.choice(sorted(POSES))
    w = _log(rng, 160, 1920)
    h = max(90, int(w * rng.uniform(0.45, 0.75)))
    if kind == "frame":
        w = _log(rng, 160, 3000)
        return {"kind": kind, "pose": pose, "width": w, "height": max(90, int(w * rng.uniform(0.45, 0.6)))}
    if kind == "engine" or kind == "flight":
        return {"kind": kind, "width": w, "height": h}
    if kind == "batch":
        return {"kind": kind, "views": rng.randint(1, 12), "width": _log(rng, 320, 1600),
                "mixed": rng.random() < 0.7, "graph": rng.random() < 0.5}
    if kind == "build":
        return {"kind": kind, "views": rng.randint(1, 8), "columns": _log(rng, 1, 128)}
    if kind == "rays":
        if rng.random() < 0.3:
            return {"kind": kind, "rays": _log(rng, 500, 8192), "exhaustive": True}
        return {"kind": kind, "rays": _log(rng, 1000, 200000), "exhaustive": False}
    if kind == "serve":
        return {"kind": kind, "sessions": rng.randint(1, 8), "width": _log(rng, 640, 1920)}
    return {"kind": kind, "pose": pose, "width": w, "height": h}


def _world(seed, k=0):
    """The world seed of an input (exact as a float32 camera word)."""
    return (WORLD_SEED + 7919 * int(seed) + 104729 * k) & 0xFFFFFF


def _view(name, seed, width, height, k=0):
    (x, z), pos, yaw, pitch = POSES[name]
    v = View(width, height)
    v.set_pose(_world(seed, k), (x, 0, z, 0), pos, yaw, pitch)
    return v


def _mixed_specs(case, seed):
    """Views as many users would have them: 16:9 of log-uniform width up to the
    case's (the same widths for every seed), any 64-bit lot address, 1.5-300 m
    high, looking anywhere from 45 degrees down to 10 up."""
    sizes = np.random.default_rng(999)
    rng = np.random.default_rng(1000 + int(seed))
    specs = []
    for _ in range(case["views"]):
        w = int(round(case["width"] / 6.0 * 6.0 ** sizes.random()))
        origin = [int(x) for x in rng.integers(0, 2**32, size=4, dtype=np.uint64)]
        pos = (float(rng.uniform(-18, 18)), float(rng.uniform(1.5, 300.0)), float(rng.uniform(-18, 18)))
        yaw, pitch = math.radians(rng.uniform(0, 360)), math.radians(rng.uniform(-45, 10))
        specs.append((w, max(16, int(round(w * 9 / 16))), int(rng.integers(0, 1 << 24)), origin, pos, yaw, pitch))
    return specs


def _batch_views(case, seed):
    if not case["mixed"]:
        names = list(POSES)
        h = int(round(case["width"] * 9 / 16))
        return [_view(names[k % 6], seed, case["width"], h, k // 6) for k in range(case["views"])]
    views = []
    for w, h, world, origin, pos, yaw, pitch in _mixed_specs(case, seed):
        v = View(w, h)
        v.set_pose(world, origin, pos, yaw, pitch)
        views.append(v)
    return views


def _frame_of(v):
    return [v.Hit, v.Surface, v.Linear, v.History, v.Pixels]


def _prepare_serve(case, seed):
    rng = np.random.default_rng(3000 + int(seed))
    widths = [max(64, int(case["width"] * f)) for f in (1.0, 0.48, 0.64, 1.2)]
    sizes = [(w, int(round(w * 9 / 16))) for w in (widths[i % 4] for i in range(case["sessions"]))]
    srv = Server(24 << 30, max_views=8, streams=3, tune=TUNE)
    sessions = []
    for w, h in sizes:
        world = int(rng.integers(0, 1 << 24))
        origin = [int(x) for x in rng.integers(0, 2**32, size=4, dtype=np.uint64)]
        y, yaw, pitch = float(rng.uniform(1.5, 60.0)), float(rng.uniform(0, 2 * math.pi)), float(rng.uniform(-0.25, 0.0))
        # a walk of 32 steps of half a metre, there and back
        walk = []
        for i in range(32):
            s = 0.5 * (i if i < 16 else 31 - i) - 4.0
            walk.append(Pose.make(origin, (math.sin(yaw) * s, y, math.cos(yaw) * s), yaw, pitch))
        sessions.append({"sid": srv.open(world, w, h), "walk": walk, "out": np.zeros(w * h, np.uint32)})
    for s in sessions:  # a session is resident once its first request is done
        srv.wait(srv.submit(s["sid"], s["walk"][31], 1), 600000)
    return {"kind": "serve", "server": srv, "sessions": sessions, "step": 0}


def _train(state):
    v, net = state["view"], state["net"]
    sb.call("stratum_materialStep", sb.ptr(v.World), sb.ptr(v.Origin), sb.ptr(v.C), sb.ptr(v.Hit), sb.ptr(v.Surface),
            *(sb.ptr(net[k]) for k in ("W", "M", "V", "Brain")), 0, v.width, v.height,
            torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return {"kind": kind, "view": _view(case["pose"], seed, case["width"], case["height"])}
    if kind == "engine":
        e = Engine().init(case["width"], case["height"], seed=_world(seed), exact_size=True)
        e.input[0] = 1.0  # walking forward
        return {"kind": kind, "engine": e}
    if kind == "batch":
        b = Batch(_batch_views(case, seed), TUNE)
        if case["graph"]:
            b.frame()
            b.capture()
        return {"kind": kind, "batch": b, "graph": case["graph"]}
    if kind == "flight":
        v = View(case["width"], case["height"])
        v.set_pose(_world(seed), (0xFFFFFFF0, 0, 0, 0), (0.0, 40.0, 0.0), math.pi / 2, 0.0)
        v.C[12] = 360.0  # 36 m, one lot, with every step of 0.1 s
        v.I[0] = 1.0
        b = Batch([v], TUNE)
        b.set_dt(0.1)
        return {"kind": kind, "batch": b}
    if kind == "build":
        views = [View(64, 64) for _ in range(case["views"])]
        rng = np.random.default_rng(2000 + int(seed))
        for k, v in enumerate(views):
            origin = [int(x) for x in rng.integers(0, 2**32, size=4, dtype=np.uint64)]
            sb.call("stratum_initCamera", sb.ptr(v.C), sb.ptr(v.Origin), _world(seed, k),
                    torch.cuda.current_stream().cuda_stream)
            v.Origin.copy_(torch.from_numpy(np.asarray(origin, np.uint32).view(np.int32)))
        b = Batch(views, TUNE, group_cache=0)
        b.refresh()
        return {"kind": kind, "batch": b, "words": case["columns"] * sb.WORLD_SIDE * sb.LOT_FLOATS}
    if kind == "rays":
        v = View(64, 64)
        v.set_pose(_world(seed), (0xFFFFFFF0, 0, 0, 0), (0.0, 40.0, 0.0), math.pi / 2, 0.0)
        n = case["rays"]
        rng = np.random.default_rng(4000 + int(seed))
        ro = np.stack([rng.uniform(-1000, 1000, n), rng.uniform(0.5, 100.0, n), rng.uniform(-1000, 1000, n)], 1)
        d = rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        q = np.concatenate([ro, d, np.full((n, 1), 0.0015)], 1).astype(np.float32)
        return {"kind": kind, "view": v, "rays": torch.from_numpy(q).cuda(), "exhaustive": case["exhaustive"]}
    if kind == "serve":
        return _prepare_serve(case, seed)
    v = _view(case["pose"], seed, case["width"], case["height"])
    v.frame()
    z = lambda n: torch.zeros(n, dtype=torch.float32, device="cuda")  # noqa: E731
    net = {"W": z(sb.NN_PARAMS), "M": z(sb.NN_PARAMS), "V": z(sb.NN_PARAMS), "Brain": z(32)}
    sb.call("stratum_initNeural", *(sb.ptr(net[k]) for k in ("W", "M", "V", "Brain")), int(seed) & 0xFFFF,
            torch.cuda.current_stream().cuda_stream)
    v.C[16] = 1.0  # shading uses the network once its gate has opened
    state = {"kind": kind, "view": v, "net": net}
    for i in range(160):  # frames that train, with other sampled pixels each
        v.C[6] = 4.0 * i
        _train(state)
    return state


def run(state):
    kind = state["kind"]
    if kind == "frame":
        state["view"].frame()
        return _frame_of(state["view"])
    if kind == "engine":
        e = state["engine"]
        e.frame(1 / 60)
        return [e.buffers[k] for k in ("Hit", "Surface", "Linear", "History", "Pixels", "C", "Origin")]
    if kind == "batch" or kind == "flight":
        b = state["batch"]
        if state.get("graph"):
            b.replay()
        else:
            b.frame()
        return [t for v in b.views for t in _frame_of(v)]
    if kind == "build":
        b = state["batch"]
        for v in b.views:
            v.World[: state["words"]].zero_()  # these lots are no longer described
        b.refresh()
        return [{"World": v.World, "Tags": v.Tags, "Nodes": v.Nodes} for v in b.views]
    if kind == "rays":
        return sr.trace(state["view"], state["rays"], state["exhaustive"])
    if kind == "serve":
        srv, k = state["server"], state["step"] % 32
        state["step"] += 1
        requests = [srv.submit(s["sid"], s["walk"][k], 1, s["out"]) for s in state["sessions"]]
        for r in requests:
            srv.wait(r, 60000)
        return [s["out"].view(np.uint8) for s in state["sessions"]]
    v, net = state["view"], state["net"]
    _train(state)
    sb.call("stratum_shadePixelsNeural", sb.ptr(v.World), sb.ptr(v.Origin), sb.ptr(v.C), sb.ptr(v.Hit),
            sb.ptr(v.Surface), sb.ptr(v.Linear), sb.ptr(net["W"]), sb.ptr(net["Brain"]), v.width, v.height, 0, v.height,
            torch.cuda.current_stream().cuda_stream)
    return [v.Linear, net["W"], net["M"], net["V"], net["Brain"]]


def work(case):
    """Bytes read and written once, and the reference algorithm's FP32 operations."""
    kind = case["kind"]
    if kind == "build":
        n, lots = case["views"], case["columns"] * sb.WORLD_SIDE
        return {"bytes": float(n * (TABLE_BYTES + lots * 127 * 32)),
                "flops": float(n * lots * FEATURES_PER_LOT * OPS_PER_FEATURE)}
    if kind == "rays":
        # an exhaustive ray tests every feature of each lot it crosses (about 12 of them)
        ops = 12 * FEATURES_PER_LOT * (OPS_PER_FEATURE + 30.0) if case["exhaustive"] else OPS_PER_RAY
        return {"bytes": float(case["rays"] * (28 + 32) + TABLE_BYTES), "flops": float(case["rays"]) * ops}
    if kind == "serve":
        px = sum(w * int(round(w * 9 / 16)) for w in
                 (max(64, int(case["width"] * (1.0, 0.48, 0.64, 1.2)[i % 4])) for i in range(case["sessions"])))
        return {"bytes": float(px * (PIXEL_BYTES + 4) + case["sessions"] * TABLE_BYTES), "flops": px * OPS_PER_RAY}
    if kind == "surrogate":
        px = case["width"] * case["height"]
        return {"bytes": float(px * 48 + TABLE_BYTES), "flops": px * 2600.0}
    if kind == "batch":
        if case["mixed"]:
            px = sum(w * h for w, h, *_ in _mixed_specs(case, 0))
        else:
            px = case["views"] * case["width"] * int(round(case["width"] * 9 / 16))
        return {"bytes": float(px * PIXEL_BYTES + case["views"] * TABLE_BYTES), "flops": px * OPS_PER_RAY}
    px = case["width"] * case["height"]
    return {"bytes": float(px * PIXEL_BYTES + TABLE_BYTES), "flops": px * OPS_PER_RAY}


# ---- 64-bit values ------------------------------------------------------------
def _mix(x):
    x = np.asarray(x, np.uint64) & 0xFFFFFFFF
    x ^= x >> np.uint64(16)
    x = (x * np.uint64(2146121005)) & np.uint64(0xFFFFFFFF)
    x ^= x >> np.uint64(15)
    x = (x * np.uint64(2221713035)) & np.uint64(0xFFFFFFFF)
    return x ^ (x >> np.uint64(16))


def _key(xl, xh, zl, zh, seed):
    u = np.uint64
    return _mix(xl * u(1973) + _mix(xh + u(719)) + zl * u(9277) + _mix(zh + u(173)) + u((seed * 26699) & 0xFFFFFFFF))


def _descriptors(origin, seed):
    """The lot table of a 64-bit origin in double precision: 16,384 x 16."""
    u, m = np.uint64, np.uint64(0xFFFFFFFF)
    slot = np.arange(sb.WORLD_LOTS)
    side = sb.WORLD_SIDE
    cx = (slot % side - (origin[0] & 127) + side // 2) % side - side // 2
    cz = (slot // side - (origin[2] & 127) + side // 2) % side - side // 2

    def axis(lo, hi, d):
        v = (np.uint64(lo) | (np.uint64(hi) << u(32))) + d.astype(np.int64).astype(np.uint64)
        return v & m, v >> u(32)
    xl, xh = axis(origin[0], origin[1], cx)
    zl, zh = axis(origin[2], origin[3], cz)
    key = _key(xl, xh, zl, zh, seed)
    dk = _key((xl >> u(3)) | ((xh << u(29)) & m), xh >> u(3), (zl >> u(3)) | ((zh << u(29)) & m), zh >> u(3), seed + 47)

    def part(k):
        return (_mix(key + u(k)) & u(65535)).astype(np.float64) / 65536.0
    r, density = (key & u(65535)).astype(np.float64) / 65536.0, (dk & u(65535)).astype(np.float64) / 65536.0
    kind = np.where(r > float(np.float32(0.94)), 1, 0)
    kind = np.where(r < 0.10 + density * 0.045, 3, kind)
    kind = np.where((xl & u(63)) == 28, np.where((zl & u(3)) == 0, 4, 5), kind)
    kind = np.where((key & u(255)) == 93, 2, kind)
    floors = 2 + np.floor(part(11) * 5.0)
    floors = np.where((density > float(np.float32(0.7))) & (floors < 4), 4, floors)
    storey = 3.2 + 1.15 * part(127)
    floors = np.where(kind == 2, 6, floors)
    offset = kind < 3
    turn = np.where(offset, ((key >> u(6)) & u(3)).astype(np.float64), 0.0)
    table = np.zeros((sb.WORLD_LOTS, 16))
    cols = [9.4 + 4.3 * part(31), 9.0 + 4.7 * part(83), 4.2 + floors * storey, kind, (key >> u(4)) & u(1), floors,
            part(271) * 65536.0, storey, 0.85 + 0.4 * part(317), turn, np.where(offset, (part(311) - 0.5) * 0.48, 0.0),
            np.where(offset, (part(313) - 0.5) * 0.48, 0.0), (dk >> u(18)) & u(7)]
    for i, c in enumerate(cols):
        table[:, i] = c
    table[:, 15] = 1.0
    return table


def exact(case, seed):
    """The lot descriptors in 64 bits.  Frames and rays have no such value: which
    feature a ray meets, and every hashed texture value, changes with the
    rounding of single coordinates."""
    if case["kind"] != "build":
        return None
    rng = np.random.default_rng(2000 + int(seed))
    out = []
    for k in range(case["views"]):
        origin = [int(x) for x in rng.integers(0, 2**32, size=4, dtype=np.uint64)]
        out.append({"World": _descriptors(origin, _world(seed, k)).reshape(-1), "Tags": None, "Nodes": None})
    return out
