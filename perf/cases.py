"""The work that is timed: what a program built on this package has it do, each
case one call (or one short sequence of calls) through the public entry points.

Sizes and scenes are those of the benchmark's configurations and of the tests
(`omg_audio_gb300.workloads`), from the smallest call of a game tick to the
large batches of an offline bake:

  box        one analytic shoebox, the late backend's call of a tick
  world      one source/listener pair on an uploaded world with panes, a tick
  shoebox    one 4096-ray job on a 12-triangle room (1 ms bins, 200 bounces)
  pairs      many source/listener pairs of the 40-room world, one batch
  rooms      uneven independent rooms, 3 and 8 bands, a batch kept and relaunched
  city       a large outdoor mesh, 8 bands, many rays a source
  labels     shoebox rooms with apertures: the surrogate's training labels
  dome       ambient dome fans of many listeners
  early      early reflections: chain discovery, then every source x chain pair
  query      surrogate inference, an ensemble over many rooms
  grad       one member's loss and gradients on a batch
  train      surrogate training steps of a whole ensemble
"""
import math
import os
import struct
import tempfile

import numpy as np

from omg_audio_gb300 import Context, DomeProbe, Job, MeshBuilder, TraceConfig, _lib
from omg_audio_gb300 import materials as M
from omg_audio_gb300 import workloads as W
from omg_audio_gb300.early import WorldEarly
from omg_audio_gb300.surrogate import Mlp, aperture_boxes, features, sample_rooms

BVH = {"sah": _lib.BVH_SAH, "sah3": _lib.BVH_SAH3, "lbvh": _lib.BVH_LBVH}
PRESETS = [M.CONCRETE, M.DRYWALL, M.CARPET, M.WOOD_PANEL, M.ACOUSTIC_TILE, M.BRICK]


def listed():
    return [
        # GpuLateBackend.trace: the reference's own tick constants (300 x 10 ms bins, 64 bounces, first-found rule)
        {"name": "box_tick", "kind": "box", "rays": 1024, "bins": 300, "bounces": 64},
        # GpuWorldLateBackend.trace_world: 512 rays x 8 on the reference's tree, panes as panels
        {"name": "world_tick", "kind": "world", "nx": 8, "ny": 5, "edge": 2.3, "rays": 4096, "bins": 300,
         "bounces": 64, "tie": 0, "bvh": "sah"},
        # the shoebox configuration: 10 x 7 x 4 m as 12 triangles, one listener
        {"name": "shoebox_mesh", "kind": "shoebox", "rays": 4096, "bins": 2000, "bounces": 200, "bvh": "sah3"},
        # the headline batch: 64 pairs x 4096 rays on the 40-room world
        {"name": "pairs_40rooms", "kind": "pairs", "nx": 8, "ny": 5, "edge": 2.3, "pairs": 64, "rays": 4096,
         "bins": 2000, "bounces": 200, "bvh": "sah3", "wt": False},
        # the uneven batch: lognormal triangles and rays, 3 or 8 bands, 0.5-4 s histograms
        {"name": "rooms_uneven", "kind": "rooms", "rooms": 96, "tri_median": 2000, "bounces": 200, "bvh": "sah3",
         "wt": False},
        # the city: a mesh far beyond the caches' reach of one room, 8 octave bands, 4 s at 1 ms
        {"name": "city_8band", "kind": "city", "nx": 10, "ny": 6, "sources": 16, "rays": 262144, "bins": 4000,
         "bounces": 200, "bvh": "sah3"},
        # the surrogate's labels: shoebox rooms with four apertures, 2 s at 1 ms
        {"name": "labels_box", "kind": "labels", "rooms": 256, "rays": 8192, "bins": 2000, "bounces": 200},
        # the dome fans of the headline step's listeners
        {"name": "dome_64x512", "kind": "dome", "nx": 8, "ny": 5, "edge": 2.3, "eyes": 64, "rays": 512, "tie": 1,
         "bvh": "sah3"},
        # early reflections for one listener: a 768-ray discovery and 64 sources x its chains
        {"name": "early_64src", "kind": "early", "nx": 8, "ny": 5, "edge": 2.3, "fan": 768, "sources": 64},
        # the surrogate asked for the held-out set
        {"name": "query_10k", "kind": "query", "n": 10000, "n_in": 38, "hidden": 256, "n_hidden": 4, "n_out": 192,
         "members": 4},
        # one gradient of the training batch
        {"name": "grad_4096", "kind": "grad", "n": 4096, "n_in": 38, "hidden": 256, "n_hidden": 4, "n_out": 192},
        # two epochs of the ensemble's training at the benchmark's batch
        {"name": "train_64steps", "kind": "train", "n": 131072, "batch": 4096, "epochs": 2, "n_in": 38,
         "hidden": 256, "n_hidden": 4, "n_out": 192, "members": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "world", "shoebox", "pairs", "rooms", "city", "labels", "dome", "early", "query",
                       "grad", "train"])
    c = {"kind": kind}
    if kind in ("world", "pairs", "dome", "early"):
        c.update(nx=rng.randint(2, 8), ny=rng.randint(1, 5), edge=round(rng.uniform(2.3, 6.0), 2))
    if kind == "box":
        c.update(rays=_log(rng, 256, 16384), bins=_log(rng, 100, 2000), bounces=rng.randint(16, 200))
    elif kind == "world":
        c.update(rays=_log(rng, 512, 8192), bins=_log(rng, 100, 2000), bounces=rng.randint(16, 200),
                 tie=rng.randint(0, 1), bvh=rng.choice(["sah", "sah3"]))
    elif kind == "shoebox":
        c.update(rays=_log(rng, 512, 16384), bins=_log(rng, 300, 4000), bounces=rng.randint(16, 200),
                 bvh=rng.choice(["sah", "sah3", "lbvh"]))
    elif kind == "pairs":
        c.update(pairs=_log(rng, 2, 64), rays=_log(rng, 512, 4096), bins=_log(rng, 300, 2000),
                 bounces=rng.randint(16, 200), bvh=rng.choice(["sah3", "sah3", "sah", "lbvh"]),
                 wt=rng.random() < 0.25)
    elif kind == "rooms":
        c.update(rooms=_log(rng, 4, 96), tri_median=_log(rng, 200, 4000), bounces=rng.randint(16, 200),
                 bvh=rng.choice(["sah3", "sah", "lbvh"]), wt=rng.random() < 0.25)
    elif kind == "city":
        c.update(nx=rng.randint(2, 10), ny=rng.randint(2, 6), sources=_log(rng, 1, 16), rays=_log(rng, 4096, 262144),
                 bins=_log(rng, 500, 4000), bounces=rng.randint(16, 200), bvh=rng.choice(["sah3", "sah3", "lbvh"]))
    elif kind == "labels":
        c.update(rooms=_log(rng, 8, 256), rays=_log(rng, 512, 8192), bins=_log(rng, 300, 2000),
                 bounces=rng.randint(16, 200))
    elif kind == "dome":
        c.update(eyes=_log(rng, 1, 256), rays=rng.choice([384, 512]), tie=rng.randint(0, 1),
                 bvh=rng.choice(["sah3", "sah"]))
    elif kind == "early":
        c.update(fan=_log(rng, 256, 4096), sources=_log(rng, 1, 100))
    else:
        c.update(n_in=rng.choice([38, 38, 24, 6]), hidden=rng.choice([256, 256, 128, 64]),
                 n_hidden=rng.randint(2, 4), n_out=rng.choice([192, 192, 64, 3]))
        if kind == "query":
            c.update(n=_log(rng, 1, 32768), members=rng.randint(1, 4))
        elif kind == "grad":
            c.update(n=128 * _log(rng, 1, 64))
        else:
            c.update(batch=rng.choice([512, 1024, 4096]), epochs=rng.randint(1, 3), members=rng.randint(1, 4))
            c["n"] = c["batch"] * rng.randint(4, 32) + rng.randint(0, 100)
    return c


# ------------------------------------------------------------------ states
def _cfg(case, **kw):
    """The benchmark's constants: 1 ms bins, energy floor 1e-6, the near-tie rule."""
    d = dict(n_bins=case.get("bins", 2000), bin_dt=0.001, max_time=case.get("bins", 2000) * 0.001,
             max_bounces=case.get("bounces", 200), energy_floor=1e-6, tie_mode=1, timeout_ms=60000,
             tri_test=1 if case.get("wt") else 0)
    d.update(kw)
    return TraceConfig(**d)


def _tick_cfg(case):
    """The reference's tick: 10 ms bins, floor 1e-7, its first-found rule unless asked otherwise."""
    return TraceConfig(n_bins=case["bins"], bin_dt=0.01, max_time=case["bins"] * 0.01, max_bounces=case["bounces"],
                       tie_mode=case.get("tie", 0), timeout_ms=60000)


def _upload(ctx, rec, nb, bvh):
    mb = MeshBuilder()
    rec.replay(mb)
    return ctx.upload_builder(mb, nb, BVH[bvh])


def _world(case, seed, n_pairs=64):
    return W.multiroom(seed=1000 + seed, nx=case["nx"], ny=case["ny"], n_pairs=n_pairs, wall_max_edge=case["edge"])


def _in_room(rng, size):
    return tuple(float(rng.uniform(0.2 * s, 0.8 * s)) for s in size)


def _box_state(case, seed, rng):
    size = (float(rng.uniform(4, 16)), float(rng.uniform(4, 12)), float(rng.uniform(2.5, 6)))
    walls = [PRESETS[int(rng.integers(len(PRESETS)))] for _ in range(6)]
    return {"ctx": Context(_tick_cfg(case)), "size": size, "walls": walls, "src": _in_room(rng, size),
            "lis": _in_room(rng, size), "rays": case["rays"], "seed": int(rng.integers(1 << 31))}


def _world_state(case, seed, rng):
    w = _world(case, seed, 2)
    ctx = Context(_tick_cfg(case))
    src, lis = w.pairs[seed % 2]
    return {"ctx": ctx, "scene": _upload(ctx, w.recorder, 3, case["bvh"]), "src": src, "lis": lis,
            "panels": w.panels, "rays": case["rays"], "seed": int(rng.integers(1 << 31))}


def _shoebox_state(case, seed, rng):
    b = W.shoebox12(seed=seed)
    ctx = Context(_cfg(case))
    return {"ctx": ctx, "scene": _upload(ctx, b.recorder, 3, case["bvh"]), "src": b.src, "lis": b.lis, "panels": (),
            "rays": case["rays"], "seed": int(rng.integers(1 << 31))}


def _pairs_state(case, seed, rng):
    w = _world(case, seed, case["pairs"])
    ctx = Context(_cfg(case))
    scene = _upload(ctx, w.recorder, 3, case["bvh"])
    jobs = [Job(src, lis, case["rays"], seed=int(rng.integers(1 << 31)), scene=scene, panel_offset=0,
                n_panels=len(w.panels)) for src, lis in w.pairs]
    return {"ctx": ctx, "jobs": jobs, "panels": w.panels, "scene": scene}


def _rooms_state(case, seed, rng):
    # the same rooms for every seed (their histogram lengths are the outputs' sizes), other poses and rays
    rooms = W.room_batch(seed=case["rooms"], n_rooms=case["rooms"], tri_median=float(case["tri_median"]))
    ctx = Context(_cfg(case, n_bands=8))
    jobs = [Job(_in_room(rng, r.size), _in_room(rng, r.size), r.n_rays, seed=int(rng.integers(1 << 31)),
                scene=_upload(ctx, r.recorder, r.n_bands, case["bvh"]), n_bands=r.n_bands, n_bins=r.n_bins,
                max_time=r.max_time) for r in rooms]
    return {"ctx": ctx, "batch": ctx.batch(jobs), "jobs": jobs}


def _city_state(case, seed, rng):
    c = W.city(seed=seed, nx=case["nx"], ny=case["ny"], n_sources=case["sources"], n_dome=1)
    ctx = Context(_cfg(case, n_bands=8))
    scene = _upload(ctx, c.recorder, 8, case["bvh"])
    jobs = [Job(tuple(map(float, s)), tuple(map(float, l)), case["rays"], seed=int(rng.integers(1 << 31)),
                scene=scene) for s, l in zip(c.sources, c.listeners)]
    return {"ctx": ctx, "batch": ctx.batch(jobs), "jobs": jobs, "scene": scene}


def _labels_state(case, seed, rng):
    rooms = sample_rooms(case["rooms"], seed)
    mn, mx, _ = aperture_boxes(rooms.size)
    jobs, panels = [], []
    for i in range(len(rooms)):
        walls = [M.Material(tuple(float(a) for a in rooms.alpha[i, w]), 0.1, (0.0,) * 3) for w in range(6)]
        off = len(panels)
        for k in range(4):
            op = float(rooms.openness[i, k])
            panels.append((tuple(mn[i, k]), tuple(mx[i, k]), M.Material((op,) * 3, 0.0, (0.0,) * 3)))
        jobs.append(Job(tuple(rooms.src[i]), tuple(rooms.lis[i]), case["rays"], seed=int(rng.integers(1 << 31)),
                        box_size=tuple(rooms.size[i]), box_walls=walls, panel_offset=off, n_panels=4))
    return {"ctx": Context(_cfg(case)), "jobs": jobs, "panels": panels}


def _dome_state(case, seed, rng):
    w = _world(case, seed, case["eyes"])
    ctx = Context(_cfg({}, tie_mode=case["tie"]))
    scene = _upload(ctx, w.recorder, 3, case["bvh"])
    return {"ctx": ctx, "probe": DomeProbe(ctx, scene, w.glass, n_fan=512), "eyes": w.listeners,
            "rays": case["rays"], "scene": scene}


def _early_state(case, seed, rng):
    w = _world(case, seed, case["sources"])
    ctx = Context(TraceConfig(timeout_ms=60000))
    scene = _upload(ctx, w.recorder, 3, "sah")
    early, lis = WorldEarly(ctx, scene), w.pairs[0][1]
    # the chain table as earlier calls filled it: the direct path and the chains of six rotations
    table = sorted({c for rot in range(6) for c in early.discover(lis, 768, rot)})
    table = (table * (1 + 399 // len(table)))[:399] if table else []
    return {"ctx": ctx, "early": early, "scene": scene, "lis": lis, "fan": case["fan"], "rot": 6 + int(rng.integers(6)),
            "table": [((_lib.NO_SURF,) * 3, 0)] + table, "sources": [(8 * i, s) for i, (s, _) in enumerate(w.pairs)],
            "extras": [(a, b, m.transmission) for a, b, m in w.panels]}


def _dims(case):
    d = [case["n_in"]] + [case["hidden"]] * case["n_hidden"] + [case["n_out"]]
    return [(d[k + 1], d[k]) for k in range(len(d) - 1)]


def _weights(case, seed):
    """He-normal layers and small biases, and the standardization of the inputs and outputs, as a trained net has."""
    rng = np.random.default_rng(77 + seed)
    norm = [rng.normal(0, 1, case["n_in"]), rng.uniform(0.5, 2, case["n_in"]), rng.uniform(-40, 0, case["n_out"]),
            rng.uniform(5, 15, case["n_out"])]
    nets = []
    for _ in range(case.get("members", 1)):
        nets.append([(rng.normal(0, math.sqrt(2.0 / i), (o, i)).astype(np.float32),
                      rng.normal(0, 0.05, o).astype(np.float32)) for o, i in _dims(case)])
    return [v.astype(np.float32) for v in norm], nets


def _net(ctx, case, seed):
    """A checkpoint of those weights, loaded as a program loads its trained surrogate."""
    norm, nets = _weights(case, seed)
    w = np.concatenate([v.ravel() for v in norm] + [v.ravel() for net in nets for wb in net for v in wb])
    m = np.zeros(2 * (len(w) - sum(len(v) for v in norm)) + 1, np.float32)
    fd, path = tempfile.mkstemp(suffix=".surrogate")
    try:
        with os.fdopen(fd, "wb") as fh:
            fh.write(Mlp.MAGIC)
            fh.write(struct.pack("<6I2Q", case["n_in"], case["hidden"], case["n_hidden"], case["n_out"], len(nets), 1,
                                 len(w), len(m)))
            fh.write(w.astype(np.float32).tobytes())
            fh.write(m.tobytes())
        return Mlp.load(ctx, path)
    finally:
        os.unlink(path)


def _query_x(case, seed):
    norm, _ = _weights(case, seed)
    rng = np.random.default_rng(seed)
    return (rng.normal(0, 1, (case["n"], case["n_in"])) * norm[1] + norm[0]).astype(np.float32)


def _grad_xy(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (case["n"], case["n_in"])).astype(np.float32)
    return x, rng.normal(0, 1, (case["n"], case["n_out"])).astype(np.float32)


def _train_state(case, seed, rng):
    ctx = Context(TraceConfig(timeout_ms=60000))
    net = Mlp(ctx, case["n_in"], case["hidden"], case["n_hidden"], case["n_out"], case["members"], seed=1 + seed)
    if case["n_in"] == 38:
        x = features(sample_rooms(case["n"], seed))
    else:
        x = rng.normal(0, 1, (case["n"], case["n_in"])).astype(np.float32)
    # decay curves: dB against time at rates that the inputs set, with the labels' noise
    k = np.abs(x[:, :3]).mean(1, keepdims=True) + 0.2
    y = np.maximum(-60.0 * np.linspace(0.02, 1, case["n_out"])[None, :] / k, -60.0) + rng.normal(0, 0.3, (case["n"],
                                                                                                        case["n_out"]))
    net.set_data(x, y.astype(np.float32))
    return {"ctx": ctx, "net": net, "epochs": case["epochs"], "batch": case["batch"]}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "query":
        ctx = Context(TraceConfig(timeout_ms=60000))
        s = {"ctx": ctx, "net": _net(ctx, case, seed), "x": _query_x(case, seed)}
    elif kind == "grad":
        ctx = Context(TraceConfig(timeout_ms=60000))
        x, y = _grad_xy(case, seed)
        s = {"ctx": ctx, "net": _net(ctx, case, seed), "x": x, "y": y}
    else:
        s = {"box": _box_state, "world": _world_state, "shoebox": _shoebox_state, "pairs": _pairs_state,
             "rooms": _rooms_state, "city": _city_state, "labels": _labels_state, "dome": _dome_state,
             "early": _early_state, "train": _train_state}[kind](case, seed, rng)
    s["kind"] = kind
    return s


# ------------------------------------------------------------------ one pass
def _one(e, rv):
    return {"bins": e.bins, "dirs": e.dirs, "rt60": rv.rt60, "level": rv.level, "fit": rv.rt60_fit,
            "segments": rv.segments}


def _many(res):
    """A batch's echograms are views of two arrays: those, and the jobs' reverb."""
    e = res[0][0]
    return {"bins": e.bins.base, "dirs": e.dirs.base, "rt60": np.concatenate([rv.rt60 for _, rv in res]),
            "level": np.concatenate([rv.level for _, rv in res]),
            "fit": np.concatenate([rv.rt60_fit for _, rv in res]),
            "segments": np.array([rv.segments for _, rv in res], np.int64)}


def run(s):
    kind = s["kind"]
    if kind == "box":
        return _one(*s["ctx"].trace_box(s["size"], s["walls"], s["src"], s["lis"], s["rays"], seed=s["seed"]))
    if kind in ("world", "shoebox"):
        return _one(*s["ctx"].trace_world(s["scene"], s["src"], s["lis"], s["rays"], s["panels"], seed=s["seed"]))
    if kind in ("pairs", "labels"):
        return _many(s["ctx"].trace_batch(s["jobs"], s["panels"]))
    if kind in ("rooms", "city"):
        s["batch"].launch()
        return _many(s["batch"].read())
    if kind == "dome":
        r = s["probe"].sample(s["eyes"], n_rays=s["rays"])
        return {"energy": r["energy"], "dir": r["dir"], "raw": r["raw"], "escape": r["escape"], "ray_tp": r["ray_tp"],
                **r["segments"]}
    if kind == "early":
        found = s["early"].discover(s["lis"], s["fan"], s["rot"])
        rec = s["early"].solve(s["sources"], s["table"], s["lis"], s["extras"])
        chains = np.full((3 * s["fan"], 4), -1, np.int64)   # as many as one call can find
        if found:
            chains[:len(found)] = [c + (o,) for c, o in found]
        return {"chains": chains, "delay": rec["delay_s"], "dir": rec["dir"], "gains": rec["gains"],
                "key": rec["key"], "valid": rec["valid"]}
    if kind == "query":
        mean, spread = s["net"].query(s["x"], -30.0)
        return {"mean": mean, "spread": spread}
    if kind == "grad":
        loss, g = s["net"].grad(s["x"], s["y"])
        return {"loss": loss, "grads": [v for wb in g for v in wb]}
    losses = s["net"].train(s["epochs"], s["batch"])
    return {"losses": losses, "weights": s["net"]._params(1)}


# ------------------------------------------------------------------ what a pass cannot do without
def _segments(rays, bounces):
    """Segments of `rays` rays: they end after about 50 on these workloads, or at the bounce limit."""
    return rays * min(bounces, 50)


def _trace_work(rays, bounces, prims, bands, bins, jobs):
    """Per segment: a descent (two slab tests a level, 24 operations each), two triangle tests, the shading."""
    depth = math.log2(prims + 1) if prims else 0
    flops = _segments(rays, bounces) * (48.0 * depth + (100.0 if prims else 40.0) + 60.0 + 4.0 * bands)
    return {"bytes": 112.0 * prims + 4.0 * jobs * bins * (bands + 3) + 200.0 * jobs, "flops": flops}


def _world_prims(case):
    return 31.0 * case["nx"] * case["ny"] * (9.0 / case["edge"] + 3.0) ** 2


def work(case):
    kind = case["kind"]
    if kind == "box":
        return _trace_work(case["rays"], case["bounces"], 0, 3, case["bins"], 1)
    if kind == "world":
        return _trace_work(case["rays"], case["bounces"], _world_prims(case), 3, case["bins"], 1)
    if kind == "shoebox":
        return _trace_work(case["rays"], case["bounces"], 12, 3, case["bins"], 1)
    if kind == "pairs":
        return _trace_work(case["pairs"] * case["rays"], case["bounces"], _world_prims(case), 3, case["bins"],
                           case["pairs"])
    if kind == "rooms":
        # lognormal triangles and rays (means 1.65 x the medians), 5.5 bands, 2250 bins on average
        return _trace_work(6750 * case["rooms"], case["bounces"], 1.65 * case["tri_median"], 5.5, 2250,
                           case["rooms"])
    if kind == "city":
        # rays leave for the sky after about 11 segments
        w = _trace_work(case["sources"] * case["rays"], min(case["bounces"], 11), 9700.0 * case["nx"] * case["ny"], 8,
                        case["bins"], case["sources"])
        return w
    if kind == "labels":
        return _trace_work(case["rooms"] * case["rays"], case["bounces"], 0, 3, case["bins"], case["rooms"])
    if kind == "dome":
        n, prims = case["eyes"] * case["rays"], _world_prims(case)
        return {"bytes": 112.0 * prims + n * (13.0 + 12.0), "flops": n * 4 * (48.0 * math.log2(prims + 1) + 160.0)}
    if kind == "early":
        pairs, prims = case["sources"] * 400, _world_prims(case)
        return {"bytes": 112.0 * prims + 52.0 * pairs,
                "flops": (6 * pairs + 3 * case["fan"]) * (48.0 * math.log2(prims + 1) + 100.0)}
    par = float(sum(o * i for o, i in _dims(case)))
    if kind == "query":
        return {"bytes": 4.0 * case["n"] * (case["n_in"] + case["n_out"] + 1) + 4.0 * par * case["members"],
                "flops": 2.0 * par * case["n"] * case["members"]}
    if kind == "grad":
        return {"bytes": 4.0 * case["n"] * (case["n_in"] + case["n_out"]) + 8.0 * par, "flops": 6.0 * par * case["n"]}
    steps = case["epochs"] * (case["n"] // case["batch"])
    return {"bytes": case["members"] * steps * (4.0 * case["batch"] * (case["n_in"] + case["n_out"]) + 24.0 * par),
            "flops": 6.0 * par * case["batch"] * steps * case["members"]}


# ------------------------------------------------------------------ the same in 64 bits
def _gelu(z):
    return 0.5 * z * (1.0 + np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def _gelu_grad(z):
    t = np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3))
    return 0.5 * (1 + t) + 0.5 * z * (1 - t * t) * 0.7978845608028654 * (1 + 3 * 0.044715 * z * z)


def _forward(net, a):
    zs, acts = [], [a]
    for k, (w, b) in enumerate(net):
        z = acts[-1] @ w.astype(np.float64).T + b
        zs.append(z)
        acts.append(z if k + 1 == len(net) else _gelu(z))
    return zs, acts


def exact(case, seed):
    """The network's own mathematics; traces, fans and chains follow every rounding of f32, so have no such value."""
    if case["kind"] == "query":
        norm, nets = _weights(case, seed)
        x = (_query_x(case, seed).astype(np.float64) - norm[0]) / norm[1]
        y = np.stack([_forward(n, x)[1][-1] * norm[3] + norm[2] for n in nets])
        # (the spread of a row reads a threshold on the mean: no value apart from its rounding)
        return {"mean": y.mean(0), "spread": None}
    if case["kind"] == "grad":
        _, nets = _weights(case, seed)
        x, y = (v.astype(np.float64) for v in _grad_xy(case, seed))
        zs, acts = _forward(nets[0], x)
        e = acts[-1] - y
        d, g = 2.0 * e / e.size, []
        for k in range(len(nets[0]) - 1, -1, -1):
            g = [d.T @ acts[k], d.sum(0)] + g
            if k:
                d = (d @ nets[0][k][0].astype(np.float64)) * _gelu_grad(zs[k - 1])
        return {"loss": float((e * e).mean()), "grads": g}
    return None
