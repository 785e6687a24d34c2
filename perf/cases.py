"""What this framework is timed on: the water engine's calls as a program makes them.

Every case is a plain dict; ``listed`` names the ones that are always timed and ``draw`` makes more of
the same ranges. A simulated case is an episode: the scene is put back as it was loaded (the
fluid's tables reset, the voxels the last episode changed written back), woken, ticked, and its
voxel changes are downloaded, so that every pass does the same work from the same state.

Kinds
  frame     one frame of an editor or a game: a brush stroke into a pool, the wake box around it,
            one fixed-rate update, the changes back on the host. Launches and latency.
  basin     the 64^3 basin with a falling block (the water's own unit scene).
  dam       the dam break on noise terrain; scale 1 is the 512 x 128 x 512 headline scene.
  lake      a deep walled lake drained through a hole in its floor: long pressure searches.
  ring      the streamed ring world with rain emitters every 4 ticks; scale 1 is 9 x 9 chunks.
  regions   many independent regions in one batched launch; scale 1 has 64 of them.
  edits     the same with a sphere brush and a wake per region between two runs of ticks.
  brush     one large sphere stroke into a lake (displacing its water), no ticks.
  save      what a save file takes of a running scene: all partial volumes, the FIFO, a box of it.
  propose   the wake-proposal network over the feature rows of a world's bricks.
  train     its gradients on a batch of labelled rows.
"""
import ctypes
import importlib

import numpy as np
import torch

vf = importlib.import_module("voxelforge-rustrewrite_b200")
proposal = importlib.import_module("voxelforge-rustrewrite_b200.proposal")

STONE, WATER = vf.STONE, vf.WATER
CAP = 50000  # cells a tick drains at most
ROWS = 1 << 17  # rows an episode's list comes back in, padded with -1 (lists of another length are another shape)


def listed():
    return [
        # a player digs in a shallow pool: the smallest call, one tick
        {"name": "frame", "kind": "frame", "side": 64, "radius": 3},
        # the unit scene: a block falls and spreads, the first levelling pass
        {"name": "basin", "kind": "basin", "block": 16, "ticks": 11},
        # a quarter-size dam break, the size of one streamed neighbourhood
        {"name": "dam quarter", "kind": "dam", "scale": 0.25, "ticks": 16},
        # the headline scene from its first tick: the cap binds first, then the channel flows
        {"name": "dam", "kind": "dam", "scale": 1.0, "ticks": 16},
        # draining a lake: every search runs into its budgets
        {"name": "lake", "kind": "lake", "side": 48, "depth": 56, "ticks": 4},
        # the open world in rain: 50,000 cells every tick, hardly any search
        {"name": "ring rain", "kind": "ring", "scale": 1.0, "ticks": 12},
        # a server's many small worlds at once
        {"name": "regions", "kind": "regions", "scale": 0.5, "ticks": 2},
        # the same with its players' brushes
        {"name": "regions edits", "kind": "edits", "scale": 0.25, "ticks": 2},
        # one big stroke, thousands of cells in order
        {"name": "brush", "kind": "brush", "radius": 9},
        # saving a running dam break
        {"name": "save", "kind": "save", "scale": 0.5, "ticks": 30},
        # scoring every brick of the ring world
        {"name": "propose", "kind": "propose", "rows": 23137},
        # a training batch of the default schedule
        {"name": "train", "kind": "train", "rows": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frame", "basin", "dam", "dam", "lake", "ring", "regions", "edits", "brush", "save", "propose", "train"])
    if kind == "frame":
        return {"kind": kind, "side": rng.randrange(40, 121), "radius": rng.randrange(1, 5)}
    if kind == "basin":
        return {"kind": kind, "block": rng.randrange(6, 17), "ticks": rng.randrange(3, 12)}
    if kind == "dam":
        return {"kind": kind, "scale": round(0.125 * 8.0 ** rng.random(), 4), "ticks": rng.randrange(5, 17)}
    if kind == "lake":
        return {"kind": kind, "side": rng.randrange(20, 49), "depth": rng.randrange(8, 57), "ticks": rng.randrange(1, 5)}
    if kind == "ring":
        return {"kind": kind, "scale": round(0.12 + 0.5 * rng.random(), 4), "ticks": rng.randrange(5, 13)}
    if kind in ("regions", "edits"):
        return {"kind": kind, "scale": round(0.08 * 3.0 ** rng.random(), 4), "ticks": rng.randrange(1, 3)}
    if kind == "brush":
        return {"kind": kind, "radius": rng.randrange(3, 10)}
    if kind == "save":
        return {"kind": kind, "scale": round(0.125 * 4.0 ** rng.random(), 4), "ticks": rng.randrange(5, 31)}
    if kind == "propose":
        return {"kind": kind, "rows": _log(rng, 33, 23137)}
    return {"kind": kind, "rows": _log(rng, 33, 8192)}


# ---------------------------------------------------------------------------------- the scenes
def _pool(side, depth, top):
    """A walled stone basin with water of `depth` on its floor."""
    w = vf.World(side, top, side)
    w.fill_box(0, 0, 0, side - 1, 3, side - 1, STONE)
    for box in ((0, 0, side - 1, 1), (0, side - 2, side - 1, side - 1), (0, 0, 1, side - 1), (side - 2, 0, side - 1, side - 1)):
        w.fill_box(box[0], 4, box[1], box[2], top - 1, box[3], STONE)
    w.fill_box(2, 4, 2, side - 3, 3 + depth, side - 3, WATER)
    return w


def _sphere(cx, cy, cz, r):
    """The cells of a sphere brush, z then y then x."""
    a = np.arange(-r, r + 1)
    z, y, x = np.meshgrid(a, a, a, indexing="ij")
    keep = x * x + y * y + z * z <= r * r
    return np.stack([x[keep] + cx, y[keep] + cy, z[keep] + cz], 1).astype(np.int32)


def _rows_of(a, rows=ROWS):
    out = np.full((rows,) + a.shape[1:], -1, a.dtype)
    out[: min(len(a), rows)] = a[:rows]
    return out


class Scene:
    """A loaded world, its handle, and what puts it back: the materials it was loaded with."""

    def __init__(self, world, wakes, stream=None):
        self.sim = vf.FluidSim(world, stream=stream)
        self.wakes = [tuple(map(int, b)) for b in wakes]
        self.info = world.info
        self.grid, self.bricks, _ = world.arrays()
        self.changed = None

    def materials(self, xyz):
        i = self.info
        x, y, z = xyz[:, 0].astype(np.int64), xyz[:, 1].astype(np.int64), xyz[:, 2].astype(np.int64)
        bx, bz = x >> 3, z >> 3
        if i.ring_w:
            bx, bz = bx & (i.bricks_x - 1), bz & (i.bricks_z - 1)
        v = self.grid[(bz * i.bricks_y + (y >> 3)) * i.bricks_x + bx].astype(np.int64)
        inside = np.maximum(v - 256, 0) * 512 + (z & 7) * 64 + (y & 7) * 8 + (x & 7)
        return np.where(v < 256, v, self.bricks[inside]).astype(np.int32)

    def put_back(self):
        sim = self.sim
        sim.reset()
        if self.changed is not None and len(self.changed):
            e = np.ascontiguousarray(self.changed)
            e[:, 3] = self.materials(e)
            p = e.ctypes.data_as(ctypes.POINTER(vf.Voxel))
            sim._check(vf.lib().vf_fluid_apply_voxel_edits(sim.h, p, len(e)), "apply_voxel_edits")

    def wake(self):
        for b in self.wakes:
            self.sim.wake(*b)

    def changes(self):
        """The episode's voxel changes, by (z, y, x): the download's own order carries no meaning."""
        c = self.sim.download_changes()
        c = c[np.lexsort((c[:, 0], c[:, 1], c[:, 2]))]
        self.changed = c.copy()
        return c

    def end(self, rows=ROWS):
        """What the host takes back: the changes, and the digests of all voxels, partial volumes, the
        FIFO and the seeds."""
        c, st = self.changes(), self.sim.stats()
        count = np.array([len(c), st.active_count, st.seed_count, st.partial_count, st.last_tick_cells, st.level_round], np.int64)
        return {"changes": _rows_of(c, rows), "count": count, "digest": np.array(self.sim.digest(), np.uint64).view(np.int64)}


def _dam(scale, rng):
    wl = vf.Workload(2, scale, 1)
    w = wl.world(0)
    n = w.info.nx
    for _ in range(6):  # boulders and holes along the channel, so that no two inputs are alike
        r = rng.uniform(2.0, 5.0)
        w.fill_sphere(rng.uniform(0, n), rng.uniform(26, 50), n / 2 + rng.uniform(-10, 10), r, int(rng.choice([0, STONE])))
    w.compact()
    return w, wl.wakes(0)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"case": case}
    if kind == "frame":
        n, r = case["side"], case["radius"]
        w = _pool(n, 6, 24)
        s["scene"] = Scene(w, [])
        c = rng.integers(2 + r, n - 2 - r, 2)
        s["cells"] = _sphere(int(c[0]), int(rng.integers(5, 10)), int(c[1]), r)
        lo, hi = s["cells"].min(0) - 1, s["cells"].max(0) + 1
        s["scene"].wakes = [(int(lo[0]), int(lo[1]), int(lo[2]), int(hi[0]), int(hi[1]), int(hi[2]))]
        s["box"] = (0, 0, 0, n, 24, n)
    elif kind == "basin":
        b = case["block"]
        w = vf.World(64, 64, 64)
        w.fill_box(0, 0, 0, 63, 3, 63, STONE)
        for box in ((6, 6, 7, 57), (56, 6, 57, 57), (6, 6, 57, 7), (6, 56, 57, 57)):
            w.fill_box(box[0], 4, box[1], box[2], 63, box[3], STONE)
        x, z, y = (int(v) for v in rng.integers((9, 9, 20), (55 - b, 55 - b, 62 - b)))
        w.fill_box(x, y, z, x + b - 1, y + b - 1, z + b - 1, WATER)
        w.compact()
        s["scene"] = Scene(w, [(x - 1, y - 1, z - 1, x + b, y + b, z + b)])
        s["box"] = (0, 0, 0, 64, 64, 64)
    elif kind == "dam":
        w, wakes = _dam(case["scale"], rng)
        s["scene"] = Scene(w, wakes)
        n = w.info.nx
        s["box"] = (0, 28, n // 2 - 8, n, 24, 16)
    elif kind == "lake":
        n, d = case["side"], case["depth"]
        w = _pool(n, d, d + 16)
        h = max(2, n // 6)
        x, z = (int(v) for v in rng.integers(3, n - 3 - h, 2))
        w.fill_box(x, 0, z, x + h - 1, 3, z + h - 1, 0)
        s["scene"] = Scene(w, [(0, 0, 0, n - 1, d + 15, n - 1)])
        s["box"] = (0, 0, 0, n, d + 16, n)
    elif kind == "ring":
        wl = vf.Workload(4, case["scale"], seed)
        s["scene"] = Scene(wl.world(0), wl.wakes(0))
        s["rain"] = wl.emitters(0)
        s["every"] = wl.emit_every
    elif kind in ("regions", "edits"):
        wl = vf.Workload(3 if kind == "regions" else 5, case["scale"], seed)
        s["stream"] = torch.cuda.Stream()
        s["scenes"] = [Scene(wl.world(r), wl.wakes(r), s["stream"].cuda_stream) for r in range(wl.regions)]
        s["batch"] = vf.Batch([c.sim for c in s["scenes"]])
        if kind == "edits":
            s["edits"] = [wl.edit(r, 9) for r in range(wl.regions)]
    elif kind == "brush":
        n, r = 64, case["radius"]
        w = _pool(n, 2 * r + 2, 2 * r + 24)
        s["scene"] = Scene(w, [])
        c = rng.integers(3 + r, n - 3 - r, 2)
        s["cells"] = _sphere(int(c[0]), 4 + r + int(rng.integers(0, 3)), int(c[1]), r)
        s["box"] = (0, 0, 0, n, 2 * r + 24, n)
    elif kind == "save":
        w, wakes = _dam(case["scale"], rng)
        s["scene"] = Scene(w, wakes)
        s["scene"].wake()
        s["scene"].sim.tick(case["ticks"])
        n = w.info.nx
        s["box"] = (0, 20, n // 2 - 32, n, 48, 64)
    else:
        n = case["rows"]
        p, x, y = _rows(n, seed)
        s["mlp"] = proposal.MLP(seed=1)
        s["mlp"].set_params(p)
        s["x"] = torch.from_numpy(x).cuda()
        s["y"] = torch.from_numpy(y).cuda()
    return s


def _rows(n, seed):
    """Network parameters and feature rows like those of a world's bricks: fractions in 0..1, half of
    them zero, a few signed flux terms, a constant; labels for a third of the rows."""
    rng = np.random.default_rng(seed)
    p = np.zeros(6337, np.float32)
    p[0:2048] = rng.normal(0, 0.25, 2048)
    p[2048:2112] = rng.normal(0, 0.05, 64)
    p[2112:6208] = rng.normal(0, 0.18, 4096)
    p[6208:6272] = rng.normal(0, 0.05, 64)
    p[6272:6336] = rng.normal(0, 0.2, 64)
    x = rng.random((n, 32)) * (rng.random((n, 32)) < 0.5)
    x[:, 19:26] = rng.normal(0, 0.1, (n, 7))
    x[:, 30] = 1.0
    y = (rng.random(n) < 1 / 3).astype(np.float32)
    return p, x.astype(np.float16), y


# -------------------------------------------------------------------------------------- a pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "propose":
        return s["mlp"].forward(s["x"], torch)
    if kind == "train":
        return s["mlp"].grads(s["x"], s["y"])
    if kind == "save":
        sim = s["scene"].sim
        xyz, vol = sim.partials()
        fifo, seeds = sim.queue()
        mat, part = sim.export_box(*s["box"])
        return {"cells": _rows_of(xyz), "volumes": _rows_of(vol), "fifo": _rows_of(fifo), "seeds": _rows_of(seeds, 4096), "materials": mat, "partials": part}
    if kind in ("regions", "edits"):
        scenes, batch = s["scenes"], s["batch"]
        for c in scenes:
            c.put_back()
            c.wake()
        batch.tick_async(case["ticks"])
        if kind == "edits":
            batch.sync()
            for c, e in zip(scenes, s["edits"]):
                c.sim.apply_brush(e[0], e[1])
                c.sim.wake(*map(int, e[2]))
            batch.tick_async(case["ticks"])
        batch.sync()
        ends = [c.end(1 << 14) for c in scenes]
        return {k: np.concatenate([e[k] for e in ends]) for k in ends[0]}
    scene = s["scene"]
    sim = scene.sim
    scene.put_back()
    if kind == "brush":
        n = sim.apply_brush(s["cells"], STONE)
        out = dict(scene.end(), written=n)
    elif kind == "frame":
        sim.apply_brush(s["cells"], 0)
        sim.apply_brush(s["cells"][: len(s["cells"]) // 2], STONE)
        scene.wake()
        sim.update(0.05)
        out = scene.end()
    elif kind == "ring":
        cells, amount = s["rain"]
        scene.wake()
        for t in range(0, case["ticks"], s["every"]):
            sim.emit(cells, amount)
            sim.tick(min(s["every"], case["ticks"] - t))
        out = scene.end()
    else:
        scene.wake()
        sim.tick(case["ticks"])
        out = scene.end()
    if "box" in s:
        out["materials"], out["partials"] = sim.export_box(*s["box"])
    return out


def work(case):
    """Bytes: a cell-step reads and writes a cell once (10 B: a material byte and a f32 volume each way);
    a search or fill entry reads one (5 B); what is exported is read and written once."""
    k = case["kind"]
    if k == "frame":
        cells = 4.2 * case["radius"] ** 3
        return {"bytes": 10 * 2 * cells + 2 * 5 * case["side"] ** 2 * 24, "flops": 0}
    if k == "basin":
        return {"bytes": 10.0 * case["block"] ** 3 * 1.6 * case["ticks"] + 10 * 64**3, "flops": 0}
    if k == "dam":
        n = 512 * case["scale"]
        return {"bytes": 10.0 * (min(CAP, n * 10 * 98) * min(case["ticks"], 12) + 40 * n * max(0, case["ticks"] - 12)) + 10 * n * 24 * 16, "flops": 0}
    if k == "lake":
        return {"bytes": (10.0 * min(CAP, case["side"] ** 2 * case["depth"]) + 5 * 512 * 2000) * case["ticks"], "flops": 0}
    if k == "ring":
        return {"bytes": 10.0 * CAP * min(1.0, 5 * case["scale"] ** 2) * case["ticks"], "flops": 0}
    if k in ("regions", "edits"):
        regions = 64 if case["scale"] >= 1 else max(2, round(64 * case["scale"]))
        return {"bytes": (10.0 * 25000 * min(1.0, 8 * case["scale"] ** 2)) * regions * case["ticks"] * (2 if k == "edits" else 1), "flops": 0}
    if k == "brush":
        return {"bytes": 4.2 * case["radius"] ** 3 * (1 + 27 / 8 + 2 * 10) + 10 * 64 * 64 * (2 * case["radius"] + 24), "flops": 0}
    if k == "save":
        n = 512 * case["scale"]
        return {"bytes": 10 * n * 48 * 64 + n * 40 * 32.0, "flops": 0}
    n = case["rows"]
    fwd = 2.0 * n * (32 * 64 + 64 * 64 + 64)
    if k == "propose":
        return {"bytes": n * 68.0 + 6337 * 4, "flops": fwd}
    return {"bytes": n * 68.0 + 6337 * 8, "flops": 3 * fwd}


def exact(case, seed):
    """The network and its mean-BCE gradient in 64 bits. The water's volumes are decided by its
    thresholds step after step in 32 bits: they have no value in 64."""
    if case["kind"] not in ("propose", "train"):
        return None
    p, x, y = _rows(case["rows"], seed)
    p, x, y = p.astype(np.float64), x.astype(np.float64), y.astype(np.float64)
    w1, b1, w2, b2, w3, b3 = p[:2048].reshape(32, 64), p[2048:2112], p[2112:6208].reshape(64, 64), p[6208:6272], p[6272:6336], p[6336]
    h1 = np.maximum(x @ w1 + b1, 0)
    h2 = np.maximum(h1 @ w2 + b2, 0)
    prob = 1 / (1 + np.exp(-(h2 @ w3 + b3)))
    if case["kind"] == "propose":
        return prob
    d = (prob - y) / len(y)
    d2 = np.outer(d, w3) * (h2 > 0)
    d1 = (d2 @ w2.T) * (h1 > 0)
    return np.concatenate([(x.T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), h2.T @ d, [d.sum()]])
