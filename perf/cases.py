"""The engine's work as its users give it: the cases whose speed is followed from change to change.

Each case is one call (or one forward / backward pair) through the public API on a mesh, batch or
scene that a program keeps, with that call's rays, points or shapes.  Meshes are the torus knots and
icospheres of the benchmark; their surface noise, and every ray, point and shape, comes from the seed.
Where a case says `tuned`, the handle carries the traversal setting and leaf layout that the autotuner
picks for that workload on this GPU; the others run a handle as it is created.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

import __graft_entry__ as _entry

pkg = _entry.load_package()
from three_mesh_bvh_b200.batched import BatchedMeshBVH  # noqa: E402

DEV = "cuda"
INF = math.inf


def listed():
    return [
        # a click in a viewer: one ray from host memory, the Intersection back on the host
        dict(name="pick_one", op="pick", tubular=400, radial=100),
        # a few thousand rays a frame (line-of-sight, brush or audio rays), near / far set, both sides
        dict(name="rays_4k", op="first", rays="box", n=4097, tubular=200, radial=25, side=2, near=1.0, far=60.0,
             tuned=False),
        # the 1,000,000-ray set on the 80,000-triangle knot, on a handle as it is created
        dict(name="rays_1m", op="first", rays="box", n=1_000_000, tubular=400, radial=100, side=0, near=0.0, far=INF,
             tuned=False),
        # incoherent rays (light transport, visibility sampling) on the 2M-triangle knot
        dict(name="incoherent_16m", op="first", rays="sphere", n=1 << 24, tubular=2000, radial=500, side=0, near=0.0,
             far=INF, tuned=True),
        # an image of the 2M-triangle knot, one ray per pixel
        dict(name="camera_16m", op="first", rays="camera", n=4096 * 4096, width=4096, tubular=2000, radial=500, side=0,
             near=0.0, far=INF, tuned=True),
        # every hit along an image's rays (thickness, x-ray views, CSG)
        dict(name="all_hits_1m", op="all", rays="camera", n=1024 * 1024, width=1024, tubular=2000, radial=500, side=2,
             near=0.0, far=INF, cap=64, tuned=True),
        # closest points of scattered samples (particles, a cloud being registered)
        dict(name="closest_100k", op="closest", points="scatter", n=100_003, tubular=400, radial=100, max=INF,
             tuned=False),
        # an unsigned distance field on a grid
        dict(name="sdf_256", op="closest", points="grid", n=256 ** 3, width=256, tubular=400, radial=100, max=5.0,
             tuned=True),
        # a BatchedMesh of uneven geometries, each with its own rays, in one launch
        dict(name="batched_128", op="batched", geometries=128, triangles=20_000, rays_most=200_000),
        # world rays against the instances of a BatchedMesh
        dict(name="instances_1m", op="scene", geometries=16, triangles=20_000, instances=512, n=1 << 20),
        # one step of fitting to a depth image: forward, then gradients of vertices and rays
        dict(name="depth_step_1m", op="depth", rays="camera", n=1024 * 1024, width=1024, tubular=2000, radial=500,
             tuned=True),
        # collision checks: which spheres and which oriented boxes touch the mesh
        dict(name="overlap_256k", op="overlap", n=1 << 18, tubular=2000, radial=500),
    ]


def draw(rng):
    """One more case of the same ranges: from one ray to 2^24, 1,000 to 2,000,000 triangles."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    radial = log_int(20, 500)
    tubular = min(2000, 4 * radial + rng.randrange(0, 9))
    mesh = dict(tubular=tubular, radial=radial)
    op = rng.choice(["pick", "first", "first", "first", "all", "closest", "closest", "batched", "scene", "depth",
                     "overlap"])
    if op == "pick":
        return dict(op=op, **mesh)
    if op in ("first", "all", "depth"):
        top = {"first": 4096, "all": 1024, "depth": 1024}[op]
        tuned = op != "first" or rng.random() < 0.5
        kind = rng.choice(["box", "sphere", "camera", "camera"]) if op == "first" else "camera"
        case = dict(op=op, rays=kind, tuned=tuned, **mesh)
        if kind == "camera":
            # the tiled ray order needs a row length that is a multiple of 16
            width = log_int(64, top) // 16 * 16 if tuned else log_int(63, top)
            case |= dict(width=width, n=width * min(top, max(1, int(width * rng.uniform(0.4, 1.0)))))
        else:
            case |= dict(n=log_int(1000, 1 << 24))
        if op != "depth":
            far = rng.choice([INF, 45.0])
            case |= dict(side=rng.choice([0, 0, 1, 2]), near=rng.choice([0.0, 0.5]), far=far)
        if op == "all":
            case |= dict(cap=rng.choice([8, 16, 64]))
        return case
    if op == "closest":
        mesh = dict(tubular=min(400, tubular), radial=min(100, radial))
        if rng.random() < 0.5:
            return dict(op=op, points="scatter", n=log_int(1000, 1 << 20), max=rng.choice([INF, 5.0]), tuned=False,
                        **mesh)
        res = log_int(24, 256) // 8 * 8
        return dict(op=op, points="grid", n=res ** 3, width=res, max=5.0, tuned=True, **mesh)
    if op == "batched":
        return dict(op=op, geometries=log_int(4, 128), triangles=log_int(1000, 20_000), rays_most=log_int(5_000, 200_000))
    if op == "scene":
        return dict(op=op, geometries=log_int(2, 16), triangles=log_int(1000, 20_000), instances=log_int(3, 512),
                    n=log_int(1000, 1 << 20))
    return dict(op=op, n=log_int(1000, 1 << 18), **mesh)


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 11)


def _unit(g, n):
    v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


@lru_cache(maxsize=2)
def _camera_dirs(width, height):
    """Directions of a pinhole camera's pixels (45 degrees vertical field of view, looking along -z)."""
    tan_half = math.tan(math.radians(45.0) / 2)
    x = ((torch.arange(width, device=DEV, dtype=torch.float64) + 0.5) / width * 2 - 1) * tan_half * (width / height)
    y = (1 - (torch.arange(height, device=DEV, dtype=torch.float64) + 0.5) / height * 2) * tan_half
    d = torch.stack([x[None, :].expand(height, width), y[:, None].expand(height, width),
                     torch.full((height, width), -1.0, device=DEV, dtype=torch.float64)], -1).reshape(-1, 3)
    return (d / d.norm(dim=1, keepdim=True)).float()


def _rays(case, seed):
    g, n = _gen(seed), case["n"]
    if case["rays"] == "camera":
        d = _camera_dirs(case["width"], n // case["width"])
        at = torch.rand(2, generator=g, device=DEV) - 0.5            # the camera moves from frame to frame
        o = torch.cat([at, torch.tensor([35.0], device=DEV)]).expand(n, 3)
        return torch.cat([o, d], 1).contiguous()
    out = torch.empty(n, 6, device=DEV)
    for k in range(0, n, 1 << 22):
        m = min(1 << 22, n - k)
        o = _unit(g, m) * 40.0
        if case["rays"] == "sphere":
            d = _unit(g, m)
        else:
            d = (torch.rand(m, 3, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * 13.0 - o
            d = d / d.norm(dim=1, keepdim=True)
        out[k:k + m] = torch.cat([o, d], 1).float()
    return out


def _knot(case, seed):
    return pkg.torus_knot(10, 3, case["tubular"], case["radial"], noise_sigma=0.02, noise_seed=int(seed))


def _points(case, seed, position):
    g, n = _gen(seed), case["n"]
    lo, hi = position.min(0), position.max(0)
    if case["points"] == "grid":
        return torch.from_numpy(pkg.grid_points(lo, hi, case["width"])).to(DEV)
    pos = torch.from_numpy(position).to(DEV)
    near = pos[torch.randint(0, pos.shape[0], (n,), generator=g, device=DEV)]
    near = near + 0.3 * torch.randn(n, 3, generator=g, device=DEV)
    lo, hi = torch.tensor(lo, device=DEV), torch.tensor(hi, device=DEV)
    far = lo + (hi - lo) * (torch.rand(n, 3, generator=g, device=DEV) * 1.1 - 0.05)
    return torch.where(torch.rand(n, 1, generator=g, device=DEV) < 0.7, near, far).contiguous()


def _pick_ray(seed, geo):
    rng = np.random.default_rng(int(seed))
    tri = geo.position[geo.index.reshape(-1, 3)[rng.integers(0, geo.triangle_count)].astype(np.int64)]
    o = rng.normal(size=3)
    o = (o / np.linalg.norm(o) * 40.0).astype(np.float32)
    d = tri.mean(0) - o
    return o, (d / np.linalg.norm(d)).astype(np.float32)


def _shapes(case, seed, position):
    """Spheres (centre, radius) and oriented boxes (bvhc_intersects_box rows) in the mesh's box."""
    g, n = _gen(seed), case["n"]
    lo = torch.tensor(position.min(0), device=DEV)
    ext = torch.tensor(position.max(0), device=DEV) - lo
    radius = torch.exp(torch.rand(n, 1, generator=g, device=DEV) * math.log(200.0)) * 0.01
    spheres = torch.cat([lo + torch.rand(n, 3, generator=g, device=DEV) * ext, radius], 1).contiguous()
    q = torch.randn(n, 4, generator=g, device=DEV)
    x, y, z, w = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    boxes = torch.zeros(n, 24, device=DEV)
    half = torch.rand(n, 3, generator=g, device=DEV) * 0.95 + 0.05
    boxes[:, 0:3], boxes[:, 4:7] = -half, half
    boxes[:, 8], boxes[:, 9], boxes[:, 10] = 1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)
    boxes[:, 12], boxes[:, 13], boxes[:, 14] = 2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)
    boxes[:, 16], boxes[:, 17], boxes[:, 18] = 2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)
    boxes[:, 20:23] = lo + torch.rand(n, 3, generator=g, device=DEV) * ext
    boxes[:, 23] = 1
    return spheres, boxes


def _geometries(case, seed):
    geoms, _, _, _ = pkg.batched_scene(case["geometries"], (200, case["triangles"]), (1_000, 2_000), seed=int(seed),
                                       make_rays=False)
    return geoms


def _batched_rays(case, seed):
    """Each geometry's rays, log-uniform in number (the case's own), drawn as the 1,000,000-ray set's."""
    rng = np.random.default_rng(case["geometries"])
    counts = np.exp(rng.uniform(math.log(1_000), math.log(case["rays_most"]), case["geometries"])).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    return _rays(dict(rays="box", n=int(off[-1])), seed), off


def _instances(case, seed):
    rng = np.random.default_rng(int(seed) + 9)
    k = case["instances"]
    q = rng.normal(size=(k, 4))
    x, y, z, w = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    s = rng.uniform(0.5, 2.0, k)
    m = np.zeros((k, 16))
    m[:, 0], m[:, 1], m[:, 2] = s * (1 - 2 * (y * y + z * z)), s * 2 * (x * y + w * z), s * 2 * (x * z - w * y)
    m[:, 4], m[:, 5], m[:, 6] = s * 2 * (x * y - w * z), s * (1 - 2 * (x * x + z * z)), s * 2 * (y * z + w * x)
    m[:, 8], m[:, 9], m[:, 10] = s * 2 * (x * z + w * y), s * 2 * (y * z - w * x), s * (1 - 2 * (x * x + y * y))
    m[:, 12:15] = rng.uniform(-400, 400, (k, 3))
    m[:, 15] = 1
    return rng.integers(0, case["geometries"], k).astype(np.uint32), m


def _world_rays(case, seed):
    g, n = _gen(seed), case["n"]
    o = _unit(g, n) * 1000.0
    d = (torch.rand(n, 3, generator=g, device=DEV, dtype=torch.float64) * 2 - 1) * 400.0 - o
    return torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).float()


# ------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------

def _tune(bvh, case):
    """The autotuner's picks on this GPU: leaf layout 4; camera rays warp-cooperative over child pairs in
    8-row tiles; incoherent ones persistent over four-child records behind the root-box pre-pass;
    grids warp-cooperative in 4-row tiles."""
    if case["op"] == "closest":
        bvh.set_traversal(closest=1, occupancy=2, tile=case["width"], tile_rows=4)
        return
    if case["op"] == "all":
        bvh.set_traversal(all=1, occupancy=2, tile=case["width"], tile_rows=8)
        return
    bvh.set_leaf_size(4)
    if case["rays"] == "camera":
        bvh.set_traversal(persistent=2, order=0, occupancy=2, tile=case["width"], tile_rows=8)
    else:
        bvh.set_traversal(persistent=1, order=1, refill=32, occupancy=2, compact=1, wide=1)


def prepare(case, seed):
    op = case["op"]
    s = {"case": case, "op": op}
    if op in ("batched", "scene"):
        geoms = _geometries(case, seed)
        batch = BatchedMeshBVH(geoms, {"strategy": pkg.SAH})
        batch.set_leaf_size(4)
        s["batch"] = batch
        if op == "batched":
            batch.set_traversal(persistent=1, order=1, refill=32, occupancy=2, wide=1)
            s["rays"], s["offsets"] = _batched_rays(case, seed)
        else:
            geometry, matrices = _instances(case, seed)
            s["scene"] = batch.instances(geometry, matrices)
            s["rays"] = _world_rays(case, seed)
        return s
    geo = _knot(case, seed)
    if op == "pick":
        s["ray"] = _pick_ray(seed, geo)
    bvh = s["bvh"] = pkg.MeshBVH(geo, {"strategy": pkg.SAH, "deviceBuild": True})
    bvh._device_mesh()
    if case.get("tuned"):
        _tune(bvh, case)
    if op in ("first", "all", "depth"):
        s["rays"] = _rays(case, seed)
    if op == "all":
        n, cap = case["n"], case["cap"]
        s["out"] = (torch.zeros(n, dtype=torch.int32, device=DEV),
                    torch.zeros((n, cap, 8), dtype=torch.float32, device=DEV))
    if op == "closest":
        s["points"] = _points(case, seed, geo.position)
    if op == "depth":
        s["grad_distance"], s["grad_barycoord"] = _upstream(case, seed)
        bvh._gradients_ready()
    if op == "overlap":
        s["spheres"], s["boxes"] = _shapes(case, seed, geo.position)
    return s


def _upstream(case, seed):
    g = _gen(int(seed) + 1)
    return (torch.randn(case["n"], generator=g, device=DEV),
            torch.randn(case["n"], 3, generator=g, device=DEV))


def _hit_fields(h):
    """A record tensor's columns by name (views)."""
    return {"face": h.view(torch.int32)[..., 0], "distance": h[..., 1], "point": h[..., 2:5], "barycoord": h[..., 5:8]}


def run(s):
    case, op = s["case"], s["op"]
    if op == "pick":
        hit = s["bvh"].raycastFirst(s["ray"])
        return {"face": hit.faceIndex, "distance": np.float32(hit.distance), "point": hit.point.astype(np.float32),
                "barycoord": hit.barycoord.astype(np.float32), "normal": hit.normal.astype(np.float32),
                "uv": hit.uv.astype(np.float32)}
    if op == "first":
        return _hit_fields(s["bvh"].raycast_first_batch(s["rays"], case["side"], case["near"], case["far"]))
    if op == "all":
        counts, hits = s["bvh"].raycast_batch(s["rays"], case["side"], case["near"], case["far"], cap=case["cap"],
                                              out=s["out"])
        return {"counts": counts, **_hit_fields(hits)}
    if op == "closest":
        r = s["bvh"].closest_point_batch(s["points"], 0.0, case["max"])
        return {"face": r.view(torch.int32)[:, 0], "distance": r[:, 1], "point": r[:, 2:5]}
    if op == "batched":
        return _hit_fields(s["batch"].raycast_first(s["rays"], s["offsets"]))
    if op == "scene":
        hits, inst = s["scene"].raycast_first(s["rays"])
        return {"instance": inst, **_hit_fields(hits)}
    if op == "depth":
        hits = s["bvh"].raycast_first_batch(s["rays"])
        gv, go, gd = s["bvh"].raycast_first_backward(s["rays"], hits, s["grad_distance"], s["grad_barycoord"])
        return {"grad_vertices": gv, "grad_origins": go, "grad_directions": gd, **_hit_fields(hits)}
    return {"spheres": s["bvh"].intersects_sphere_batch(s["spheres"]), "boxes": s["bvh"].intersects_box_batch(s["boxes"])}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------

def work(case):
    """Bytes: queries in, results out, the triangles (36 B) and their boxes (32 B a node, two nodes a
    leaf of ten) once each, where that many queries can touch them all.  Flops: the boxes and the
    triangle or two that even a perfect descent tests."""
    op = case["op"]
    if op in ("batched", "scene"):
        mean = (case["triangles"] - 200) / math.log(case["triangles"] / 200)     # log-uniform sizes
        tris = case["geometries"] * mean
        n = case["n"] if op == "scene" else case["geometries"] * (case["rays_most"] - 1000) / math.log(
            case["rays_most"] / 1000)
    else:
        tris = 2 * case["tubular"] * case["radial"]
        n = case.get("n", 1)
    depth = max(1.0, math.log2(max(2.0, tris / 10)))
    per = {"pick": 56, "first": 56, "batched": 56, "closest": 32, "scene": 60, "overlap": 16 + 96 + 2}.get(op)
    if op == "all":
        per = 24 + 4 + 4 * 32
    if op == "depth":
        per = 24 + 32 + 32 + 24 + 16 + 24
    flops = n * (2 * depth * 25 + 2 * 60)
    mesh = min(tris * 42.4, n * (64 * depth + 72))
    return {"bytes": float(n * per + mesh + (12 * tris / 2 if op == "depth" else 0)), "flops": float(flops)}


# ------------------------------------------------------------------------------------------
# the same results in 64 bits: a breadth-first walk of (query, node) pairs in torch
# ------------------------------------------------------------------------------------------

class _Tree:
    """Triangles in Morton order under an implicit tree of eight children a node."""

    def __init__(self, tri):
        c = tri.mean(1)
        lo, hi = c.amin(0), c.amax(0)
        q = ((c - lo) / (hi - lo).clamp_min(1e-300) * 1023).long().clamp(0, 1023)
        code = torch.zeros(tri.shape[0], dtype=torch.int64, device=tri.device)
        for b in range(10):
            for a in range(3):
                code |= ((q[:, a] >> b) & 1) << (3 * b + a)
        self.ids = code.argsort()
        self.tri = tri[self.ids]
        lo, hi = self.tri.amin(1), self.tri.amax(1)
        self.levels = [(lo, hi)]
        while lo.shape[0] > 8:
            pad = -lo.shape[0] % 8
            lo = torch.cat([lo, lo[-1:].expand(pad, 3)]).view(-1, 8, 3).amin(1)
            hi = torch.cat([hi, hi[-1:].expand(pad, 3)]).view(-1, 8, 3).amax(1)
            self.levels.append((lo, hi))

    def top(self, n):
        k = self.levels[-1][0].shape[0]
        return (torch.arange(n, device=DEV).repeat_interleave(k), torch.arange(k, device=DEV).repeat(n))

    def below(self, query, node, level):
        node = (node[:, None] * 8 + torch.arange(8, device=DEV)).reshape(-1)
        query = query.repeat_interleave(8)
        keep = node < self.levels[level][0].shape[0]
        return query[keep], node[keep]


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


def _first_exact(tree, rays, side, near, far):
    """Nearest hit of every ray: (triangle row or -1, t), rows of tree.tri."""
    n = rays.shape[0]
    row = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    t_out = torch.full((n,), INF, dtype=torch.float64, device=DEV)
    for k in range(0, n, 1 << 17):
        r = rays[k:k + (1 << 17)].double()
        o, d = r[:, :3], r[:, 3:]
        q, node = tree.top(r.shape[0])
        for level in range(len(tree.levels) - 1, -1, -1):
            lo, hi = tree.levels[level]
            t0, t1 = (lo[node] - o[q]) / d[q], (hi[node] - o[q]) / d[q]
            keep = torch.minimum(t0, t1).amax(1) <= torch.maximum(t0, t1).amin(1).clamp_min(0) * (1 + 1e-9)
            keep &= torch.maximum(t0, t1).amin(1) >= 0
            q, node = q[keep], node[keep]
            if level:
                q, node = tree.below(q, node, level - 1)
        a, b, c = tree.tri[node].unbind(1)
        e1, e2, oa, dd = b - a, c - a, o[q] - a, d[q]
        nn = _cross(e1, e2)
        N, U, V = _dot(dd, nn), _dot(dd, _cross(oa, e2)), _dot(dd, _cross(e1, oa))
        s = N.sign()
        W = N - U - V
        ok = (N != 0) & (s * U >= 0) & (s * V >= 0) & (s * W >= 0) & (-s * _dot(oa, nn) >= 0)
        ok &= N < 0 if side == 0 else (N > 0 if side == 1 else ok)
        t = -_dot(oa, nn) / N
        dist = t * dd.norm(dim=1)
        ok &= (dist >= near) & (dist <= far)
        q, node, t = q[ok], node[ok], t[ok]
        best = torch.full((r.shape[0],), INF, dtype=torch.float64, device=DEV).scatter_reduce_(0, q, t, "amin")
        win = t == best[q]
        row[k:k + r.shape[0]][q[win]] = node[win]
        t_out[k:k + r.shape[0]] = best
    return row, t_out


def _fields_exact(tri, rays, row, t):
    """distance, point, barycoord of the nearest hits (differentiable), a miss as the engine writes it."""
    hit = (row >= 0).nonzero()[:, 0]
    a, b, c = tri[row[hit]].unbind(1)
    o, d = rays[hit, :3], rays[hit, 3:]
    e1, e2, q = b - a, c - a, o - a
    nn = _cross(e1, e2)
    N, U, V = _dot(d, nn), _dot(d, _cross(q, e2)), _dot(d, _cross(e1, q))
    tt = -_dot(q, nn) / N
    return hit, tt * d.norm(dim=1), o + tt[:, None] * d, torch.stack([(N - U - V) / N, U / N, V / N], 1)


def _place(n, hit, distance, point, bary):
    out = {"face": None, "distance": torch.full((n,), INF, dtype=torch.float64, device=DEV),
           "point": torch.zeros(n, 3, dtype=torch.float64, device=DEV),
           "barycoord": torch.zeros(n, 3, dtype=torch.float64, device=DEV)}
    out["distance"][hit], out["point"][hit], out["barycoord"][hit] = distance, point, bary
    return out


def _closest_exact(tree, pts):
    n = pts.shape[0]
    point = torch.empty(n, 3, dtype=torch.float64, device=DEV)
    for k in range(0, n, 1 << 15):
        p = pts[k:k + (1 << 15)].double()
        m = p.shape[0]
        q, node = tree.top(m)
        for level in range(len(tree.levels) - 1, -1, -1):
            lo, hi = tree.levels[level]
            near = (torch.maximum(lo[node] - p[q], p[q] - hi[node])).clamp_min(0).square().sum(1)
            far = torch.maximum(hi[node] - p[q], p[q] - lo[node]).square().sum(1)
            most = torch.full((m,), INF, dtype=torch.float64, device=DEV).scatter_reduce_(0, q, far, "amin")
            keep = near <= most[q] * (1 + 1e-12)
            q, node = q[keep], node[keep]
            if level:
                q, node = tree.below(q, node, level - 1)
        a, b, c = tree.tri[node].unbind(1)
        ab, ac, bc, pp = b - a, c - a, c - b, p[q]
        nn = _cross(ab, ac)

        def on(x, e):
            return x + e * (_dot(pp - x, e) / _dot(e, e)).clamp(0, 1)[:, None]

        best, d2 = on(a, ab), None
        d2 = (pp - best).square().sum(1)
        for x, e in ((a, ac), (b, bc)):
            c2 = on(x, e)
            e2 = (pp - c2).square().sum(1)
            best, d2 = torch.where((e2 < d2)[:, None], c2, best), torch.minimum(e2, d2)
        h = _dot(pp - a, nn) / _dot(nn, nn)
        f = pp - h[:, None] * nn
        u, v = _dot(_cross(f - a, ac), nn), _dot(_cross(ab, f - a), nn)
        inside = (u >= 0) & (v >= 0) & (u + v <= _dot(nn, nn))
        best, d2 = torch.where(inside[:, None], f, best), torch.where(inside, (pp - f).square().sum(1), d2)
        least = torch.full((m,), INF, dtype=torch.float64, device=DEV).scatter_reduce_(0, q, d2, "amin")
        win = d2 == least[q]
        point[k:k + m][q[win]] = best[win]
    return {"face": None, "distance": (point - pts.double()).norm(dim=1), "point": point}


def _triangles(geo):
    return torch.from_numpy(geo.position).to(DEV).double()[torch.from_numpy(geo.index.astype(np.int64)).to(DEV).view(-1, 3)]


def exact(case, seed):
    op = case["op"]
    if op in ("all", "overlap") or (op == "closest" and (case["max"] != INF or case["n"] > 1 << 21)):
        # hits come in the tree's order; overlaps are whole numbers; what lies beyond a finite maximum
        # distance depends on the tree's boxes
        return None
    if op == "scene":
        geometry, mats = _instances(case, seed)
        tris = [_triangles(g) for g in _geometries(case, seed)]
        m = torch.from_numpy(mats).to(DEV).view(-1, 4, 4)             # rows: the matrix's columns
        world = torch.cat([tris[g] @ m[j, :3, :3] + m[j, 3, :3] for j, g in enumerate(geometry)])
        rays = _world_rays(case, seed).double()
        tree = _Tree(world)
        row, t = _first_exact(tree, rays, 0, 0.0, INF)
        return {"instance": None, **_place(case["n"], *_fields_exact(tree.tri, rays, row, t))}
    if op == "batched":
        rays, off = _batched_rays(case, seed)
        parts = []
        for k, geo in enumerate(_geometries(case, seed)):
            r = rays[int(off[k]):int(off[k + 1])].double()
            tree = _Tree(_triangles(geo))
            row, t = _first_exact(tree, r, 0, 0.0, INF)
            parts.append(_place(r.shape[0], *_fields_exact(tree.tri, r, row, t)))
        return {"face": None, **{f: torch.cat([p[f] for p in parts]) for f in ("distance", "point", "barycoord")}}
    geo = _knot(case, seed)
    if op == "closest":
        return _closest_exact(_Tree(_triangles(geo)), _points(case, seed, geo.position))
    if op == "pick":
        o, d = _pick_ray(seed, geo)
        rays = torch.from_numpy(np.concatenate([o, d])[None]).to(DEV).double()
        tree = _Tree(_triangles(geo))
        row, t = _first_exact(tree, rays, 0, 0.0, INF)
        r = _place(1, *_fields_exact(tree.tri, rays, row, t))
        vid = torch.from_numpy(geo.index.astype(np.int64)).to(DEV).view(-1, 3)[tree.ids[row]]
        w = r["barycoord"][:, :, None]
        normal = (torch.from_numpy(geo.normal).to(DEV).double()[vid] * w).sum(1)
        normal = torch.where(_dot(normal, rays[:, 3:])[:, None] > 0, -normal, normal)
        uv = (torch.from_numpy(geo.uv).to(DEV).double()[vid] * w).sum(1)
        return {"face": None, "distance": r["distance"][0], "point": r["point"][0], "barycoord": r["barycoord"][0],
                "normal": normal[0], "uv": uv[0]}
    rays = _rays(case, seed)
    tree = _Tree(_triangles(geo))
    if op == "first":
        row, t = _first_exact(tree, rays, case["side"], case["near"], case["far"])
        out = _place(case["n"], *_fields_exact(tree.tri, rays.double(), row, t))
        return out
    row, t = _first_exact(tree, rays, 0, 0.0, INF)
    pos = torch.from_numpy(geo.position).to(DEV).double().requires_grad_()
    vid = torch.from_numpy(geo.index.astype(np.int64)).to(DEV).view(-1, 3)[tree.ids]
    o, d = rays[:, :3].double().requires_grad_(), rays[:, 3:].double().requires_grad_()
    gd, gb = (x.double() for x in _upstream(case, seed))
    hit = (row >= 0).nonzero()[:, 0]
    a, b, c = pos[vid[row[hit]]].unbind(1)
    e1, e2, q, dh = b - a, c - a, o[hit] - a, d[hit]
    nn = _cross(e1, e2)
    N, U, V = _dot(dh, nn), _dot(dh, _cross(q, e2)), _dot(dh, _cross(e1, q))
    dist = -_dot(q, nn) / N * dh.norm(dim=1)
    bary = torch.stack([(N - U - V) / N, U / N, V / N], 1)
    ((dist * gd[hit]).sum() + (bary * gb[hit]).sum()).backward()
    fields = _place(case["n"], hit, dist.detach(), (o[hit] + (dist / dh.norm(dim=1))[:, None] * dh).detach(), bary.detach())
    return {"grad_vertices": pos.grad, "grad_origins": o.grad, "grad_directions": d.grad, **fields}
