"""The calls that programs make of this library, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program has in hand
before the call (scene, tape, pools, buffers, camera), ``run`` makes the call
through the public classes (``frep.Voxelizer``, ``Raytracer``,
``AnimatedVoxelizer``, ``CompactTree``, ``Batch``, ``Server``, ``Context``) and
returns its outputs. Scenes are the library's own seeded generators
(``frep.scenes``), grids and image sizes those of its benchmark, its tests and
the reference's demo, plus odd ones of the same ranges.

Hit records are returned as depth and normal (float32), level, cell and DDA
step count; the node number of a hit is left out for device trees, whose nodes
are numbered in the order in which warps claim them (compact trees have one
numbering, so theirs is returned).

Kinds:

* ``frame``    one scene voxelized and rendered (an interactive edit, a frame
               of an animation without reuse, one request on its own);
* ``render``   a voxelized scene rendered again (a moving camera; with
               ``samples`` > 1 the temporal multi-sample image);
* ``compact``  a voxelized tree made compact and rendered (before it is saved);
* ``animated`` the next frame of an animation, with reuse of the last one;
* ``batch``    many scenes voxelized and rendered together, one graph replay;
* ``serve``    a burst of requests to the render server, new scenes and
               resident ones, images in host memory;
* ``points``   the shape's value at many points, host arrays in and out.
"""
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("f-rep-voxel-rendering_b200"))

import frep  # noqa: E402
from frep import csg, scenes  # noqa: E402
from frep.autotune import DEFAULT_TABLE, fit_pools, load_table, size_class  # noqa: E402

ROUNDINGS = {"nearest": frep.ROUND_NEAREST, "outward": frep.ROUND_OUTWARD, "hybrid": frep.ROUND_HYBRID}


def listed():
    return [
        # The smallest call: the 16-sphere union on a 64^3 grid, 256 x 256
        # orthographic (an editor's preview; latency and launches count).
        {"name": "small_frame", "kind": "frame", "scene": "spheres", "prims": 16, "grid": "16,4", "width": 256,
         "height": 256, "rounding": "outward"},
        # One of the reference's demo shapes (sine, division, time) in its
        # main()'s five-level grid (4096^3) and its own rounding.
        {"name": "demo_frame", "kind": "frame", "scene": "ElasticCube", "prims": 0, "grid": "16,4,4,4,4", "width": 1280,
         "height": 720, "rounding": "nearest"},
        # An ordinary scene on a grid without a power of two, odd image size.
        {"name": "ragged_frame", "kind": "frame", "scene": "csg", "prims": 75, "grid": "12,20,4", "width": 999,
         "height": 563, "rounding": "outward"},
        # The large scene of the benchmark: 256 primitives, 2048^3, 1080p with
        # shadow rays, voxelized and rendered.
        {"name": "large_frame", "kind": "frame", "scene": "csg", "prims": 256, "grid": "16,16,8", "width": 1920,
         "height": 1080, "rounding": "outward"},
        # The transcendental stress scene on three levels (1024^3), 1080p.
        {"name": "stress_frame", "kind": "frame", "scene": "gyroid", "prims": 64, "grid": "16,16,4", "width": 1920,
         "height": 1080, "rounding": "outward"},
        # The same large scene seen by a moving camera: only the renderer runs.
        {"name": "large_render", "kind": "render", "scene": "csg", "prims": 256, "grid": "16,16,8", "width": 1920,
         "height": 1080, "samples": 1},
        # The temporal multi-sample image (four jittered frames and their mean).
        {"name": "temporal_render", "kind": "render", "scene": "csg", "prims": 64, "grid": "16,8,4", "width": 1280,
         "height": 720, "samples": 4},
        # Compaction of the large scene's tree, pruned, and a frame of it.
        {"name": "compact_prune", "kind": "compact", "scene": "csg", "prims": 256, "grid": "16,16,8", "width": 1920,
         "height": 1080, "prune": True},
        # The animated workload: a large static part, four moving spheres.
        {"name": "animated_frame", "kind": "animated", "prims": 256, "moving": 4, "grid": "16,16,8", "width": 1920,
         "height": 1080},
        # The batching distribution (4 to 1024 primitives, 64^3 to 1024^3) at
        # 512 x 512 with shadow rays: the throughput headline.
        {"name": "batch_128", "kind": "batch", "scenes": 128, "width": 512, "height": 512, "max_prims": 1024},
        # A serving burst: 45 of 64 requests bring a new scene, the others
        # render one of 16 resident scenes again.
        {"name": "serve_64", "kind": "serve", "requests": 64, "new": 45, "width": 512, "height": 512,
         "max_prims": 1024},
        # The shape's value at a million points (sampling a field for export).
        {"name": "points_1m", "kind": "points", "prims": 64, "points": 1000000},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "render", "compact", "animated", "batch", "serve", "points"])
    w = _log(rng, 100, 1920)
    h = max(64, min(1080, int(w * rng.uniform(0.5, 0.8))))
    grid = rng.choice(["16,8", "32,8", "16,4,4", "16,8,4", "16,16,4", "16,16,8", "32,8,4", "16,8,8", "16,4,4,4", "12,8,4", "20,12",
                       "12,12,12", "8,20,4", "24,12"])
    if kind == "frame":
        scene = rng.choice(["csg", "csg", "csg", "spheres", "gyroid", "ElasticCube", "Screw", "Morph", "TangleCube",
                            "OrganicBalls"])
        prims = _log(rng, 4, 600) if scene == "csg" else _log(rng, 4, 100)
        if scene == "gyroid":
            grid = rng.choice(["16,16", "16,16,4", "12,16,4", "16,8,4"])
        rounding = rng.choice(["outward", "outward", "nearest", "hybrid"])
        return {"kind": kind, "scene": scene, "prims": prims, "grid": grid, "width": w, "height": h,
                "rounding": rounding}
    if kind == "render":
        return {"kind": kind, "scene": rng.choice(["csg", "csg", "spheres"]), "prims": _log(rng, 8, 400), "grid": grid,
                "width": w, "height": h, "samples": rng.choice([1, 1, 2, 5])}
    if kind == "compact":
        return {"kind": kind, "scene": "csg", "prims": _log(rng, 8, 400), "grid": grid, "width": w, "height": h,
                "prune": rng.random() < 0.5}
    if kind == "animated":
        return {"kind": kind, "prims": _log(rng, 8, 400), "moving": rng.randint(1, 8), "grid": grid, "width": w,
                "height": h}
    if kind == "batch":
        return {"kind": kind, "scenes": _log(rng, 2, 120), "width": min(w, 512), "height": min(h, 512),
                "max_prims": _log(rng, 64, 1024)}
    if kind == "serve":
        n = _log(rng, 2, 64)
        return {"kind": kind, "requests": n, "new": max(1, int(n * rng.uniform(0.3, 0.9))), "width": min(w, 512),
                "height": min(h, 512), "max_prims": _log(rng, 64, 1024)}
    return {"kind": kind, "prims": _log(rng, 4, 100), "points": _log(rng, 1000, 1000000)}


# ---- inputs ---------------------------------------------------------------------

def _dims(text):
    return [int(d) for d in text.split(",")]


def _orbit(rng, distance, fov=60.0):
    return scenes.orbit_camera(rng, distance, fov)


def _scene(case, seed):
    """(tape, low vertex, world size, camera, time, shadow mask) of a single-scene case."""
    rng = np.random.default_rng(seed)
    dims = _dims(case["grid"])
    kind = case.get("scene", "csg")
    n = case["prims"]
    time = 0.0
    if case["kind"] == "animated":
        sc = scenes.animated_csg(n, case["moving"], seed, dims)
        cam = _orbit(rng, 3.9)
    elif kind == "spheres":
        sc = scenes.spheres_union(n, seed, case["width"], case["height"])
        cam = sc.camera
    elif kind == "csg":
        sc = scenes.random_csg(n, seed, dims)
        cam = _orbit(rng, 3.9)
    elif kind == "gyroid":
        sc = scenes.stress_gyroid(n, seed, grid_dims=dims)
        time = float(rng.uniform(0.0, 0.3))
        cam = _orbit(rng, 4.2)
    else:  # the reference's demo shapes over [-20, 20]^3
        shape = scenes.DEMO_SHAPES[kind](0)
        sc = scenes.Scene(kind, shape, dims, (-20.0, -20.0, -20.0), 40.0)
        time = float(rng.uniform(0.0, 6.0))
        cam = frep.Camera(position=(0.0, float(rng.uniform(-4.0, 4.0)), 40.0), forward=(0.0, 0.0, -1.0),
                          initial_up=(0.0, 1.0, 0.0), fov_deg=45.0)
    return frep.Tape(sc.shape), sc.low_vertex, sc.world_size, cam, time, sc.shadow_mask


def _buffers(h, w, hits):
    rgba = torch.empty((h, w, 4), dtype=torch.uint8, device="cuda")
    rec = torch.empty((h, w, 8), dtype=torch.int32, device="cuda") if hits else None
    return rgba, rec


def _hits(rec, node=False):
    out = {"depth": rec.view(torch.float32)[..., 0], "normal": rec.view(torch.float32)[..., 1:4], "level": rec[..., 4],
           "cell": rec[..., 6], "steps": rec[..., 7]}
    if node:
        out["node"] = rec[..., 5]
    return out


def _batch_tapes(rng, n, max_prims, structures):
    """n scenes of the batching distribution: primitive counts log-uniform in
    [4, max_prims], effective resolutions 64 to 1024, every scene with constants
    of its own. `structures` of them are built, the others are variations of
    these (as the server's load generator makes its scenes)."""
    k = min(n, structures)
    wide = []
    for i in range(k):
        prims = int(round(4 * (max_prims / 4) ** ((i + rng.random()) / k)))
        wide.append(frep.Tape(scenes.random_csg(prims, int(rng.integers(1 << 30))).shape).wide())
    res = [scenes.BATCH_RESOLUTIONS[(i // k + i) % len(scenes.BATCH_RESOLUTIONS)] for i in range(n)]
    tapes = [scenes.jitter_tape(wide[i % k], rng) for i in range(n)]
    table = load_table(DEFAULT_TABLE)
    grids, cells = [], []
    for t, r in zip(tapes, res):
        c = table.get(f"{r}:{size_class(t.n_instr)}")
        grids.append(tuple(c.dims) if c else scenes.DEFAULT_BRANCHING[r])
        cells.append(c.point_cells_per_lane if c else 0)
    return tapes, grids, cells


LOW, WORLD = (-1.25, -1.25, -1.25), 2.5  # the batch scenes' box


def prepare(case, seed):
    kind = case["kind"]
    ctx = frep.Context(0, hbm_budget_bytes=48 << 30)
    s = {"case": case, "ctx": ctx}
    rng = np.random.default_rng(seed)
    if kind == "points":
        centers = rng.uniform(-1.0, 1.0, (case["prims"], 3)).astype(np.float32)
        radii = rng.uniform(0.1, 0.3, case["prims"]).astype(np.float32)
        shape = None
        for c, r in zip(centers, radii):
            ball = csg.Sphere(csg.Vector3(float(c[0]), float(c[1]), float(c[2])), float(r))
            shape = ball if shape is None else csg.Union(shape, ball)
        s["tape"] = frep.Tape(shape)
        s["xyzt"] = _points(rng, case["points"])
        return s
    w, h = case["width"], case["height"]
    if kind in ("batch", "serve"):
        lights = frep.Lights(shadow_mask=1)
        s["lights"] = lights
        if kind == "batch":
            n = case["scenes"]
            tapes, grids, cells = _batch_tapes(rng, n, case["max_prims"], 16)
            pools = fit_pools(ctx, tapes, grids, LOW, WORLD)
            trees = [frep.VoxelStorage(g, LOW, WORLD, node_words=p.node_words, tape_words=p.tape_words,
                                       point_cells_per_lane=k).init(ctx, t)
                     for t, g, k, p in zip(tapes, grids, cells, pools)]
            s["batch"] = frep.Batch(ctx, trees)
            s["cameras"] = [_orbit(rng, 4.1) for _ in range(n)]
            s["sizes"] = [(w, h)] * n
            s["rgba"] = torch.empty((n, h, w, 4), dtype=torch.uint8, device="cuda")
            s["hits"] = torch.empty((n, h, w, 8), dtype=torch.int32, device="cuda")
            s["frames"], s["records"] = list(s["rgba"]), list(s["hits"])
            return s
        n, new = case["requests"], case["new"]
        old = 16
        tapes, grids, cells = _batch_tapes(rng, new + old, case["max_prims"], 16)
        pools = fit_pools(ctx, tapes, grids, LOW, WORLD)
        srv = frep.Server(ctx, hbm_budget_bytes=24 << 30, lights=lights)
        s["server"] = srv
        s["scenes"] = [(t, g, LOW, WORLD, p.node_words, p.tape_words, k)
                       for t, g, k, p in zip(tapes, grids, cells, pools)]
        resident = [srv.add_scene(*a) for a in s["scenes"][new:]]
        s["scenes"] = s["scenes"][:new]
        # request i: a new scene (index) or a resident one (its id)
        order = rng.permutation(n)
        plan = [("new", int(i)) if i < new else ("old", resident[int(rng.integers(old))]) for i in order]
        s["plan"] = plan
        s["cameras"] = [_orbit(rng, 4.1) for _ in range(n)]
        s["images"] = torch.empty((n, h, w, 4), dtype=torch.uint8, pin_memory=True)
        for k, sid in enumerate(resident):  # resident before the burst, as after earlier requests
            srv.submit(sid, s["cameras"][k % n], 0.0, w, h, s["images"][k % n])
            srv.drain()
        return s
    tape, low, world, cam, time, shadows = _scene(case, seed)
    dims = _dims(case["grid"])
    rounding = ROUNDINGS[case.get("rounding", "outward")]
    times = [0.0, 0.31, 0.72] if kind == "animated" else [time]
    pools = fit_pools(ctx, [tape] * len(times), [dims] * len(times), low, world, tape_times=times, margin=0.1)
    # Pools from an outward voxelization; nearest rounding and the hybrid mode
    # leave the same or fewer ambiguous cells, up to a little of shape.
    nodes = max(p.node_words for p in pools) * 5 // 4
    words = max(p.tape_words for p in pools) * 5 // 4

    def storage():
        return frep.VoxelStorage(dims, low, world, rounding=rounding, node_words=nodes, tape_words=words)

    s.update(camera=cam, time=time, out=_buffers(h, w, kind in ("frame", "compact", "animated")))
    if kind == "animated":
        s["voxelizer"] = frep.AnimatedVoxelizer(ctx, storage, tape)
        s["frame"] = 0
        vs = s["voxelizer"].voxelize(0.3)  # frame 0: the one before the first pass
    else:
        vs = storage().init(ctx, tape)
        s["voxelizer"] = frep.Voxelizer(ctx, vs)
        if kind != "frame":
            s["voxelizer"].voxelize(time)
    s["voxels"] = vs
    s["raytracer"] = frep.Raytracer(ctx, vs)
    s["raytracer"].lights.shadow_mask = shadows
    return s


def _points(rng, n):
    xyzt = np.zeros((n, 4), np.float32)
    xyzt[:, :3] = rng.uniform(-1.5, 1.5, (n, 3)).astype(np.float32)
    return xyzt


# ---- one pass -------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "points":
        return s["ctx"].eval_points(s["tape"], s["xyzt"])
    w, h = case["width"], case["height"]
    if kind == "batch":
        s["batch"].run(s["cameras"], s["sizes"], s["frames"], s["records"], s["lights"], graph=True)
        return {"rgba": s["rgba"], **_hits(s["hits"])}
    if kind == "serve":
        srv = s["server"]
        ids = [srv.add_scene(*a) for a in s["scenes"]]
        reqs = [srv.submit(ids[k] if what == "new" else k, cam, 0.0, w, h, img)
                for (what, k), cam, img in zip(s["plan"], s["cameras"], s["images"])]
        states = [srv.wait(r).state for r in reqs]
        for r in reqs:
            srv.release(r)
        return {"images": s["images"], "done": sum(st == frep.REQ_DONE for st in states)}
    rt, out = s["raytracer"], s["out"]
    if kind == "frame":
        s["voxelizer"].voxelize(s["time"])
        rt.trace(s["camera"], s["time"], w, h, out=out)
        return {"rgba": out[0], **_hits(out[1])}
    if kind == "animated":
        s["frame"] += 1
        t = 0.3 + s["frame"] / 60.0
        rt.voxels = s["voxelizer"].voxelize(t)
        rt.trace(s["camera"], t, w, h, out=out)
        return {"rgba": out[0], **_hits(out[1])}
    if kind == "compact":
        tree = frep.CompactTree.from_storage(s["ctx"], s["voxels"], prune=case["prune"])
        tree.lights = rt.lights
        tree.trace(s["camera"], s["time"], w, h, out=out)
        info = tree.info()
        counts = [int(c) for c in info.node_count[:len(_dims(case["grid"]))]]
        tree.close()
        return {"rgba": out[0], **_hits(out[1], node=True), "nodes": counts}
    if case["samples"] > 1:
        rgba, layers = rt.trace_temporal(s["camera"], s["time"], w, h, case["samples"])
        return {"rgba": rgba, "layers": layers}
    rt.trace(s["camera"], s["time"], w, h, out=out)
    return {"rgba": out[0]}


# ---- work and 64-bit values --------------------------------------------------------

# Instructions per primitive of the compiled tapes (measured on the generators:
# a sphere of a plain union 14, a random CSG primitive with its operator 27, a
# gyroid's ball 25) and the surface of a scene in units of its box's face: the
# last-level nodes of a grid of N cells per axis with d^3-cell nodes are about
# `area` x (N / d)^2.
_INSTR = {"spheres": (14, 0), "csg": (27, 0), "gyroid": (25, 240)}
_AREA = {"spheres": 1.0, "csg": 2.4, "gyroid": 60.0}


def _tree(case, kind):
    """(instructions of the root tape, cells of the root, last-level nodes, words of the last level)"""
    per, base = _INSTR.get(kind, (0, 50))
    n = per * case["prims"] + base
    d = _dims(case["grid"])
    fine = int(np.prod(d))
    root = d[0] ** 3
    leaves = min(int(_AREA.get(kind, 1.0) * (fine / d[-1]) ** 2), (fine // d[-1]) ** 3)
    return n, root, leaves, leaves * (4 + d[-1] ** 3 // 16)


def work(case):
    """The tape read once, every last-level node and the images written once;
    the root tape over the root's cells (an interval instruction is at least
    two operations), a ten-instruction tape over every last-level cell, and a
    hundred operations for each pixel."""
    kind = case["kind"]
    if kind == "points":
        n = 14 * case["prims"]
        return {"bytes": 20 * case["points"] + 8 * n, "flops": n * case["points"]}
    pixels = case["width"] * case["height"]
    if kind in ("batch", "serve"):
        frames = case["scenes"] if kind == "batch" else case["requests"]
        new = case["scenes"] if kind == "batch" else case["new"]
        ratio = case["max_prims"] / 4.0
        prims = (case["max_prims"] - 4) / np.log(ratio) if ratio > 1 else 4.0
        instr = 27.0 * prims
        nodes = new * 2.4 * np.mean([(r / 6.0) ** 2 for r in scenes.BATCH_RESOLUTIONS])
        record = 36 if kind == "batch" else 4
        return {"bytes": float(new * 8 * instr + nodes * 40 + frames * pixels * record),
                "flops": float(new * 2 * instr * 4096 + nodes * 64 * 10 + frames * pixels * 100)}
    scene = case.get("scene", "csg")
    n, root, leaves, words = _tree(case, scene)
    if kind == "frame":
        return {"bytes": float(8 * n + 4 * words + 36 * pixels),
                "flops": float(2 * n * root + leaves * 640 + 100 * pixels)}
    if kind == "animated":  # the root again, a fiftieth of the tree evaluated, the rest copied
        return {"bytes": float(8 * n + 8 * words + 36 * pixels),
                "flops": float(2 * n * root + leaves * 640 / 50 + 100 * pixels)}
    if kind == "compact":
        return {"bytes": float(8 * words + 36 * pixels), "flops": float(100 * pixels)}
    return {"bytes": float(4 * pixels * (case["samples"] + (case["samples"] > 1))),
            "flops": float(100 * pixels * case["samples"])}


def exact(case, seed):
    """Values in 64 bits where a call computes plain numbers: the shape's value
    at points. (Depth, normal and colour of a pixel follow from the cell that
    its ray stops in, which has no 64-bit counterpart.)"""
    if case["kind"] != "points":
        return None
    rng = np.random.default_rng(seed)
    centers = rng.uniform(-1.0, 1.0, (case["prims"], 3)).astype(np.float32).astype(np.float64)
    radii = rng.uniform(0.1, 0.3, case["prims"]).astype(np.float32).astype(np.float64)
    p = _points(rng, case["points"])[:, :3].astype(np.float64)
    out = np.full(case["points"], np.inf)
    for c, r in zip(centers, radii):
        out = np.minimum(out, ((p - c) ** 2).sum(1) - r * r)
    return out


if __name__ == "__main__":
    for c in listed():
        print(c["name"], work(c))
    r = random.Random(1)
    for _ in range(6):
        print(draw(r))
