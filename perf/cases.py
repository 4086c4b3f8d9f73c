"""The work that users of cubiquity_gb300 have it do, as measurable cases.

A case is a volume, a set of rays and the entry point that takes them:

  call      device     intersect_volume on device tensors (the drop-in)
            batch      Batch.launch: many volumes with their own rays
            host       intersect_volume_host on page-locked host arrays
            server     Server.submit / wait: a burst of requests
            pathtrace  pathtrace: whole frames
  rays      camera     the pixels of a pinhole image of the volume
            bounce     cosine-weighted rays leaving the surfaces a camera sees
            shadow     rays towards the sun from those surfaces (hit flag only)
            collision  short rays (tmax 8..64 voxels) from points of the volume

The volume of a case is fixed (a level that the program has loaded); camera
poses, bounce directions, collision points and request streams come from the
seed.  A state owns its device copy of the volume, its rays and its outputs.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

SUN = (0.0975900073, -0.195180015, 0.975900073)  # normalize(1, -2, 10), as the demo's sun
LOD = 0.0035                                     # the demo's LOD footprint
SURFACE_FIELDS = ("hit", "distance", "material", "position", "normal", "voxel", "status")
FLOATS = {"distance": 1, "position": 3, "normal": 3}
RAY_BYTES = 32
HIT_BYTES = {"hit": 1, "distance": 4, "material": 4, "position": 12, "normal": 12, "voxel": 12, "status": 1}


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # A physics step's collision queries: the smallest call, latency and launches count.
        {"name": "collision-1k", "call": "device", "scene": "terrain", "edge_log2": 10, "rays": "collision",
         "count": 1000},
        # A preview thumbnail: a ragged image, far fewer rays than the chip holds.
        {"name": "camera-333x217", "call": "device", "scene": "spheres", "edge_log2": 8, "rays": "camera",
         "width": 333, "height": 217},
        # The small benchmark scene: camera rays on spheres-256.
        {"name": "camera-1mp-spheres", "call": "device", "scene": "spheres", "edge_log2": 8, "rays": "camera",
         "width": 1024, "height": 1024},
        # The benchmark's camera batch: a large landscape, coherent rays.
        {"name": "camera-4mp-terrain", "call": "device", "scene": "terrain", "edge_log2": 12, "rays": "camera",
         "width": 2048, "height": 2048},
        # The benchmark's bounce batch: incoherent rays from the surfaces of the landscape.
        {"name": "bounce-4m-terrain", "call": "device", "scene": "terrain", "edge_log2": 12, "rays": "bounce",
         "count": 4194304},
        # Sun shadows of a frame: no surface properties, only the hit flag, an odd number of rays.
        {"name": "shadow-1.5m-terrain", "call": "device", "scene": "terrain", "edge_log2": 11, "rays": "shadow",
         "count": 1500001},
        # A full-HD view of a big city with levels of detail.
        {"name": "lod-1080p-city", "call": "device", "scene": "city", "edge_log2": 13, "rays": "camera",
         "width": 1920, "height": 1080, "lod": True},
        # The compact node store, which a user takes to save memory.
        {"name": "bounce-1m-compact", "call": "device", "scene": "terrain", "edge_log2": 11, "rays": "bounce",
         "count": 1000000, "compact": True},
        # Many volumes with their own rays in one captured launch.
        {"name": "batch-12", "call": "batch", "volumes": 12, "edge_low": 7, "edge_high": 10, "rays_low": 16384,
         "rays_high": 524288},
        # A host program's call: rays and hits in page-locked host memory.
        {"name": "host-1m-bounce", "call": "host", "scene": "terrain", "edge_log2": 11, "rays": "bounce",
         "count": 1000003},
        # A burst of requests of several clients on resident volumes.
        {"name": "serve-24", "call": "server", "requests": 24, "rays_low": 1024, "rays_high": 65536},
        # A path-traced preview frame of a city: camera, bounce and shadow waves.
        {"name": "pathtrace-640x360", "call": "pathtrace", "scene": "city", "edge_log2": 12, "width": 640,
         "height": 360, "samples": 4, "bounces": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, most):
    n = _log_int(rng, 4096, most)
    aspect = rng.uniform(0.6, 2.4)
    w = max(16, int(math.sqrt(n * aspect)))
    return w, max(16, n // w)


def draw(rng):
    kind = rng.choice(("collision", "camera", "camera", "bounce", "bounce", "shadow", "lod", "compact", "batch", "host",
                       "server", "pathtrace"))
    if kind == "collision":
        return {"call": "device", "scene": "terrain", "edge_log2": rng.randint(7, 11), "rays": "collision",
                "count": _log_int(rng, 200, 1000000)}
    if kind in ("camera", "lod"):
        scene = rng.choice(("spheres", "terrain", "city"))
        w, h = _image(rng, 4000000)
        if rng.random() < 0.5:
            w, h = (w + 15) // 16 * 16, (h + 7) // 8 * 8  # display sizes are round
        edge = {"spheres": rng.randint(6, 9), "terrain": rng.randint(7, 11), "city": rng.randint(10, 12)}[scene]
        return {"call": "device", "scene": scene, "edge_log2": edge, "rays": "camera", "width": w, "height": h,
                "lod": kind == "lod"}
    if kind in ("bounce", "compact", "host"):
        scene = rng.choice(("terrain", "spheres"))
        edge = rng.randint(7, 11) if scene == "terrain" else rng.randint(6, 9)
        case = {"call": "host" if kind == "host" else "device", "scene": scene, "edge_log2": edge, "rays": "bounce",
                "count": _log_int(rng, 1000, 1500000 if kind == "host" else 4000000)}
        if kind == "compact":
            case["compact"] = True
        return case
    if kind == "shadow":
        return {"call": "device", "scene": "terrain", "edge_log2": rng.randint(7, 11), "rays": "shadow",
                "count": _log_int(rng, 1000, 4000000)}
    if kind == "batch":
        return {"call": "batch", "volumes": rng.randint(3, 16), "edge_low": 7, "edge_high": rng.randint(8, 10),
                "rays_low": _log_int(rng, 1024, 16384), "rays_high": _log_int(rng, 20000, 400000)}
    if kind == "server":
        return {"call": "server", "requests": rng.randint(4, 32), "rays_low": _log_int(rng, 64, 1024),
                "rays_high": _log_int(rng, 4096, 65536)}
    w, h = _image(rng, 250000)
    return {"call": "pathtrace", "scene": "city", "edge_log2": rng.randint(10, 12), "width": w, "height": h,
            "samples": rng.randint(1, 4), "bounces": rng.randint(1, 3)}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=64)
def _scene(scene: str, edge_log2: int, seed: int = 0):
    """(nodes, root) of a level: built once per process, as a program loads a file once."""
    spec = {"spheres": lambda: W.SceneSpec(cbq.SCENE_SPHERES, edge_log2, 20240607 + seed, 64),
            "terrain": lambda: W.terrain_scaled(edge_log2, 4096001 + seed),
            "city": lambda: W.SceneSpec(cbq.SCENE_CITY, edge_log2, 8192001 + seed)}[scene]()
    return spec.build()


def _pose(scene: str, edge_log2: int, seed: int):
    """A camera around the volume: the workloads' view, moved by the seed."""
    rng = random.Random(seed)
    e = float(1 << edge_log2)
    if scene == "city":
        eye, target = W.city_camera(edge_log2)
    elif scene == "terrain":
        cam = W.camera_scaled(edge_log2, 1, 1)
        eye, target = cam.eye, cam.target
    else:
        eye, target = (-0.5 * e, -0.5 * e, 1.171875 * e), (0.5 * e, 0.5 * e, 0.5 * e)
    move = lambda p, by: tuple(v + rng.uniform(-by, by) * e for v in p)  # noqa: E731
    return move(eye, 0.05), move(target, 0.05)


def _camera_rays(scene, edge_log2, width, height, seed):
    eye, target = _pose(scene, edge_log2, seed)
    return cbq.pinhole_rays(eye, target, W.TAN_30, width, height)


def _surfaces(nodes, root, scene, edge_log2, count, seed):
    """Positions and normals of the surfaces that a camera image of about `count` pixels sees."""
    side = max(32, min(2048, math.isqrt(count)))
    o, d = _camera_rays(scene, edge_log2, side, side, seed)
    dag = cbq.Dag(nodes, root)
    hits = cbq.intersect_volume(dag, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    hit = hits["hit"].bool()
    pos, nrm = hits["position"][hit], hits["normal"][hit]
    torch.cuda.synchronize()
    dag.destroy()
    return pos, nrm


def _collision_rays(edge_log2, count, seed):
    e = float(1 << edge_log2) - 1.0  # voxel centres lie at 0..edge-1: points inside the volume
    o, d = cbq.sphere_rays((0.0, 0.0, 0.0), (e, e, e / 2), count, seed)
    o[:, 3] = np.random.default_rng(seed).uniform(8.0, 64.0, count).astype(np.float32)
    return o, d


def _rays(case, seed):
    """(origin_tmax, direction) of a one-volume case, as host arrays."""
    scene, edge = case["scene"], case["edge_log2"]
    if case["rays"] == "camera":
        return _camera_rays(scene, edge, case["width"], case["height"], seed)
    if case["rays"] == "collision":
        return _collision_rays(edge, case["count"], seed)
    n = case["count"]
    pos, nrm = _surfaces(*_scene(scene, edge), scene, edge, n, seed)
    if case["rays"] == "bounce":
        return cbq.bounce_rays(pos.cpu().numpy(), nrm.cpu().numpy(), n, seed)
    pick = torch.arange(n, device="cuda") % pos.shape[0]
    o = torch.full((n, 4), math.inf, device="cuda")
    o[:, :3] = pos[pick] + 0.001 * nrm[pick]
    d = torch.zeros((n, 4), device="cuda")
    d[:, :3] = torch.tensor(SUN, device="cuda")
    return o.cpu().numpy(), d.cpu().numpy()


def _query(case):
    """Keyword arguments of the traversal calls."""
    q = {"compute_surface_properties": case["rays"] != "shadow", "use_tmax": case["rays"] == "collision"}
    if case.get("lod"):
        q["max_footprint"] = LOD
    if case["rays"] == "camera":
        q["image_width"] = case["width"]
    return q


def _fields(case):
    return ("hit",) if case.get("rays") == "shadow" else SURFACE_FIELDS


def _count(case):
    return case["count"] if "count" in case else case["width"] * case["height"]


def _batch_jobs(case, seed):
    """[(scene, edge, scene seed, rays)]: half camera rays, half collision points' rays, as the batching workload."""
    shapes = random.Random(case["volumes"] * 1009 + case["edge_high"])
    rng = random.Random(seed)
    jobs = []
    for i in range(case["volumes"]):
        scene = shapes.choice(("spheres", "terrain"))
        edge = shapes.randint(case["edge_low"], case["edge_high"])
        n = _log_int(shapes, case["rays_low"], case["rays_high"])
        side = max(8, math.isqrt(n // 2))
        o1, d1 = _camera_rays(scene, edge, side, side, rng.randrange(1 << 30))
        e = float(1 << edge) - 1.0
        o2, d2 = cbq.sphere_rays((0.0, 0.0, 0.0), (e, e, e), max(1, n - side * side), rng.randrange(1 << 30))
        jobs.append((scene, edge, i % 3, (np.concatenate([o1, o2]), np.concatenate([d1, d2]))))
    return jobs


SERVED = (("terrain", 9), ("terrain", 10), ("terrain", 10))  # resident volumes of the server


def _requests(case, seed):
    """[(volume, collision, rays)]: 70% collision rays, 30% view rays, sizes log-uniform."""
    sizes = random.Random(case["requests"] * 31 + case["rays_high"])
    rng = random.Random(seed)
    out = []
    for _ in range(case["requests"]):
        n = _log_int(sizes, case["rays_low"], case["rays_high"])
        v = sizes.randrange(len(SERVED))
        collision = sizes.random() < 0.7
        if collision:
            rays = _collision_rays(SERVED[v][1], n, rng.randrange(1 << 30))
        else:
            side = max(8, math.isqrt(n))
            rays = _camera_rays(*SERVED[v], side, side, rng.randrange(1 << 30))
        out.append((v, collision, rays))
    return out


def _pinned(a):
    """A page-locked copy of a host array (the tensor keeps it alive)."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _pinned_hits(n, fields=SURFACE_FIELDS):
    like = cbq.alloc_host_hits(1)
    kinds = {np.dtype(np.uint32): np.dtype(np.int32)}
    out = {}
    for k in fields:
        dtype = kinds.get(like[k].dtype, like[k].dtype)
        out[k] = torch.zeros((n, *like[k].shape[1:]), dtype=torch.from_numpy(np.zeros(0, dtype)).dtype).pin_memory()
    return out


def _slices(buffers, at, n, convert):
    return {k: convert(v[at:at + n]) for k, v in buffers.items()}


# ------------------------------------------------------------------ states and passes

def prepare(case, seed):
    call = case["call"]
    if call == "batch":
        jobs = _batch_jobs(case, seed)
        dags = [cbq.Dag(*_scene(s, e, k)) for s, e, k, _ in jobs]
        rays = [(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()) for _, _, _, (o, d) in jobs]
        out = cbq.alloc_hits(sum(o.shape[0] for o, _ in rays))
        views, at = [], 0
        for o, _ in rays:
            views.append(_slices(out, at, o.shape[0], lambda t: t))
            at += o.shape[0]
        batch = cbq.Batch([(g, o, d) for g, (o, d) in zip(dags, rays)], outputs=views)
        return {"call": call, "batch": batch, "dags": dags, "out": out}
    if call == "server":
        requests = _requests(case, seed)
        dags = [cbq.Dag(*_scene(s, e, k)) for k, (s, e) in enumerate(SERVED)]
        out = _pinned_hits(sum(o.shape[0] for _, _, (o, _) in requests))
        todo, at = [], 0
        for v, collision, (o, d) in requests:
            n = o.shape[0]
            po, pd = _pinned(o), _pinned(d)
            todo.append((dags[v], po, pd, cbq.Query(use_tmax=collision),
                         _slices(out, at, n, lambda t: t.numpy())))
            at += n
        server = cbq.Server(device_memory_budget=256 << 20)
        return {"call": call, "server": server, "requests": todo, "dags": dags, "out": out}
    nodes, root = _scene(case["scene"], case["edge_log2"])
    dag = cbq.Dag(nodes, root, cbq.LAYOUT_COMPACT if case.get("compact") else cbq.LAYOUT_REFERENCE)
    if call == "pathtrace":
        eye, target = _pose(case["scene"], case["edge_log2"], seed)
        return {"call": call, "dag": dag, "materials": W.city_materials(seed),
                "frame": dict(width=case["width"], height=case["height"], samples_per_pixel=case["samples"],
                              bounces=case["bounces"], eye=eye, target=target, max_footprint=LOD, seed=seed)}
    o, d = _rays(case, seed)
    state = {"call": call, "dag": dag, "query": _query(case)}
    if call == "host":
        state.update(o=_pinned(o), d=_pinned(d), out=_pinned_hits(_count(case)))
    else:
        state.update(o=torch.from_numpy(o).cuda(), d=torch.from_numpy(d).cuda(),
                     out=cbq.alloc_hits(_count(case), fields=_fields(case)))
    return state


def run(state):
    call = state["call"]
    if call == "device":
        return cbq.intersect_volume(state["dag"], state["o"], state["d"], out=state["out"], **state["query"])
    if call == "batch":
        state["batch"].launch()
        return state["out"]
    if call == "host":
        cbq.intersect_volume_host(state["dag"], state["o"].numpy(), state["d"].numpy(),
                                  out={k: v.numpy() for k, v in state["out"].items()}, **state["query"])
        return state["out"]
    if call == "server":
        server = state["server"]
        tickets = [server.submit(dag, o.numpy(), d.numpy(), query, out)[0]
                   for dag, o, d, query, out in state["requests"]]
        for t in tickets:
            server.wait(t)
        return state["out"]
    image, _ = cbq.pathtrace(state["dag"], materials=state["materials"], **state["frame"])
    return image


def work(case):
    """Rays in and hits out (the nodes that the rays meet come on top: how many depends on the
    view, and most are read from cache)."""
    call = case["call"]
    per_ray = RAY_BYTES + sum(HIT_BYTES[k] for k in _fields(case))
    if call == "pathtrace":
        # Per path and depth: an extension ray and two shadow rays, of which the frame needs the
        # image alone; counted as the rays' own 32 bytes for the camera wave and the image.
        paths = case["width"] * case["height"] * case["samples"]
        return {"bytes": paths * RAY_BYTES + case["width"] * case["height"] * 12, "flops": 0}
    if call == "batch":
        shapes = random.Random(case["volumes"] * 1009 + case["edge_high"])
        n = 0
        for _ in range(case["volumes"]):
            shapes.choice((0, 1))
            shapes.randint(case["edge_low"], case["edge_high"])
            n += _log_int(shapes, case["rays_low"], case["rays_high"])
        return {"bytes": n * per_ray, "flops": 0}
    if call == "server":
        sizes = random.Random(case["requests"] * 31 + case["rays_high"])
        n = 0
        for _ in range(case["requests"]):
            k = _log_int(sizes, case["rays_low"], case["rays_high"])
            sizes.randrange(len(SERVED))
            n += k if sizes.random() < 0.7 else max(8, math.isqrt(k)) ** 2
        return {"bytes": n * per_ray, "flops": 0}
    return {"bytes": _count(case) * per_ray, "flops": 0}


# ------------------------------------------------------------------ 64-bit answers

def _node_of_volume(nodes, root, edge_log2):
    """The node of the box [0, 2^edge_log2)^3: child 7 of the root, then children 0."""
    node, slot = root, 7
    for _ in range(31, edge_log2 - 1, -1):
        if node < 256:
            return node
        node, slot = int(nodes[8 * node + slot]), 0
    return node


def _trace64(nodes, root, edge_log2, origin_tmax, direction, max_footprint=-1.0, use_tmax=False):
    """Distance, position and normal of the first hits in 64 bits: from one leaf or empty box of
    the volume to the next along each ray, every box found from its integer corner."""
    dev = "cuda"
    table = torch.from_numpy(nodes.view(np.int32)).to(dev)
    top = _node_of_volume(nodes, root, edge_log2)
    edge = 1 << edge_log2
    total = origin_tmax.shape[0]
    res = {k: torch.zeros((total, w) if w > 1 else (total,), dtype=torch.float64, device=dev)
           for k, w in FLOATS.items()}
    for begin in range(0, total, 1 << 20):
        part = slice(begin, min(total, begin + (1 << 20)))
        o4 = torch.from_numpy(origin_tmax[part]).to(dev).double()
        d = torch.from_numpy(direction[part, :3]).to(dev).double()
        o = o4[:, :3] + 0.5
        forward = d >= 0
        inv = 1.0 / d
        ids = torch.arange(o.shape[0], device=dev)
        near = torch.where(forward, 0.0, float(edge))
        t_in = ((near - o) * inv).max(dim=1).values
        t_out = ((edge - near - o) * inv).min(dim=1).values
        start = t_in.clamp(min=0.0)
        keep = (t_in < t_out) & (t_out > 0)
        q = (o + start[:, None] * d).floor().long().clamp(0, edge - 1)
        ids, q = ids[keep], q[keep]
        while ids.numel():
            oo, ii, ff = o[ids], inv[ids], forward[ids]
            node = torch.full_like(ids, top)
            size = torch.full_like(ids, edge)
            low = torch.zeros_like(q)
            going = node >= 256
            half = edge
            while half > 1 and bool(going.any()):
                half //= 2
                bits = (q - low) >= half
                slot = bits[:, 0].long() + 2 * bits[:, 1].long() + 4 * bits[:, 2].long()
                child = table[(8 * node + slot).clamp(max=table.numel() - 1)].long()
                node = torch.where(going, child, node)
                low = torch.where(going[:, None], low + half * bits.long(), low)
                size = torch.where(going, half, size)
                going = going & (node >= 256)
                if max_footprint >= 0:
                    far = torch.where(ff, low + size[:, None], low).double()
                    going = going & (size / ((far - oo) * ii).min(dim=1).values > max_footprint)
            entry = torch.where(ff, low, low + size[:, None]).double()
            far = torch.where(ff, low + size[:, None], low).double()
            solid = node > 0
            if bool(solid.any()):
                t = (entry[solid] - oo[solid]) * ii[solid]
                dist, axis = t.max(dim=1)
                rows = ids[solid]
                if use_tmax:
                    close = dist <= o4[rows, 3]
                    rows, dist, axis = rows[close], dist[close], axis[close]
                res["distance"][part][rows] = dist
                res["position"][part][rows] = o4[rows, :3] + d[rows] * dist[:, None]
                normal = torch.zeros((rows.numel(), 3), dtype=torch.float64, device=dev)
                sign = torch.where(forward[rows], -1.0, 1.0).double()
                normal.scatter_(1, axis[:, None], sign.gather(1, axis[:, None]))
                res["normal"][part][rows] = normal
            t_exit, axis = ((far - oo) * ii).min(dim=1)
            q_next = (oo + t_exit[:, None] * d[ids]).floor().long()
            q_next = torch.minimum(torch.maximum(q_next, low), low + size[:, None] - 1)
            beyond = torch.where(ff, low + size[:, None], low - 1)
            q_next.scatter_(1, axis[:, None], beyond.gather(1, axis[:, None]))
            keep = ~solid & (q_next >= 0).all(dim=1) & (q_next < edge).all(dim=1)
            ids, q = ids[keep], q_next[keep]
    return res


def exact(case, seed):
    call = case["call"]
    if call == "pathtrace":  # a sum over random paths: another rounding takes other paths
        return None
    none = dict.fromkeys(SURFACE_FIELDS)
    if call in ("batch", "server"):
        if call == "batch":
            parts = [_trace64(*_scene(s, e, k), e, o, d) for s, e, k, (o, d) in _batch_jobs(case, seed)]
        else:
            parts = [_trace64(*_scene(*SERVED[v], v), SERVED[v][1], o, d, use_tmax=collision)
                     for v, collision, (o, d) in _requests(case, seed)]
        return {**none, **{k: torch.cat([p[k] for p in parts]) for k in FLOATS}}
    if case["rays"] == "shadow":  # hit flags only
        return None
    q = _query(case)
    found = _trace64(*_scene(case["scene"], case["edge_log2"]), case["edge_log2"], *_rays(case, seed),
                     max_footprint=q.get("max_footprint", -1.0), use_tmax=q["use_tmax"])
    return {**none, **found}
