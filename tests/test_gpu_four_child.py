"""raycastFirst over the four-child records, one lane, four and the whole warp per ray, against the per-ray child-pair
kernel byte for byte: one candidate order decides in every kernel (the nearest hit, exact ties to the
smaller record), so neither the records' shape nor the batch size may change a bit."""
import importlib
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(pkg, name):
    """(geometry, build options): a root that is a leaf within one run; one of 40 triangles (halved into
    runs under its unbounded root); leaves of 40; one root per group, with gaps; a plain tree."""
    if name == "triangle":
        return pkg.Geometry(np.array([[0, 0, 0], [4, 0, 0], [0, 4, 0]], np.float32), np.array([0, 1, 2], np.uint16)), {}
    if name == "leaf40":
        g = pkg.torus_knot(10, 3, 10, 4)
        g.index = g.index[:120]
        return g, {"maxLeafSize": 64}
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    if name == "leaves40":
        return g, {"maxLeafSize": 40}
    if name == "groups":
        g.add_group(0, 900, 0)
        g.add_group(1200, 1500, 1)
        g.add_group(3000, 600, 2)
    return g, {}


def _rays(pkg, n):
    r = np.concatenate([pkg.rays_sphere_to_box(n, seed=n), pkg.rays_incoherent(n, seed=n + 1)])[:n]
    r[::5, 3:] *= np.float32(3.5)          # directions need not be unit vectors
    r[1::7, 3] = 0.0                       # a zero component
    return r


@pytest.mark.parametrize("mesh", ["triangle", "leaf40", "leaves40", "groups", "plain"])
@pytest.mark.parametrize("n", [1, 7, 33, 24576, 24577, 131072, 131073])
def test_matches_the_per_ray_kernel(pkg, cuda, mesh, n):
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    rays = torch.from_numpy(_rays(pkg, n)).to(cuda)
    cases = [(0, 0.0, math.inf), (2, 0.0, math.inf), (1, 20.0, 45.0), (2, -5.0, 38.0)]
    for leaf in (0, 3):
        bvh.set_leaf_size(leaf)
        for compact, wide, sort in ((0, 0, 0), (1, 1, 0), (1, 0, 3)):
            for side, near, far in cases:
                bvh.set_traversal(0, 1)
                want = bvh.raycast_first_batch(rays, side, near, far)
                bvh.set_traversal(1, 1, 16, 0, compact, sort, 0, wide)
                got = bvh.raycast_first_batch(rays, side, near, far)
                bvh.synchronize()
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (leaf, compact, sort, side)
    if mesh == "groups":
        host = _rays(pkg, n)
        bvh.set_traversal(0, 1)
        want = bvh.raycast_first_batch(host, [0, 2, 1])
        bvh.set_traversal(1, 1)
        assert np.array_equal(bvh.raycast_first_batch(host, [0, 2, 1]).view(np.uint8), want.view(np.uint8))
    if mesh != "triangle":
        assert n < 33 or (want["face_index"] if mesh == "groups" else want.cpu().numpy().view(np.uint32)[:, 0]).min() < 2000


@pytest.mark.parametrize("leaf", [0, 4])
def test_parts_of_leaves_follow_a_refit(pkg, cuda, leaf):
    """Boxes of runs and of halves of leaves come from their triangles, so a refit recomputes them."""
    import torch

    g = pkg.torus_knot(10, 3, 80, 12, noise_sigma=0.05, noise_seed=4)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": 40})
    bvh.set_leaf_size(leaf)
    bvh.raycast_first_batch(pkg.rays_incoherent(8))
    rng = np.random.default_rng(5)
    bvh.refit((g.position * 1.3 + rng.normal(0, 0.4, g.position.shape)).astype(np.float32))
    for n in (3000, 140_000):
        rays = torch.from_numpy(_rays(pkg, n)).to(cuda)
        bvh.set_traversal(0, 1)
        want = bvh.raycast_first_batch(rays, 2)
        bvh.set_traversal(1, 1)
        assert torch.equal(bvh.raycast_first_batch(rays, 2).view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("mesh", ["triangle", "leaf40", "leaves40", "groups", "plain"])
@pytest.mark.parametrize("n", [1, 7, 33, 4097, 8193, 200_001])
def test_closest_matches_the_per_query_kernel(pkg, cuda, mesh, n):
    """closestPointToPoint in groups and by warps, in each query order, against the per-query kernel
    (which a minThreshold above 0 selects; 1e-30 stops at nothing else than a point on the mesh)."""
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    rng = np.random.default_rng(n)
    lo, hi = g.position.min(0) - 2, g.position.max(0) + 2
    pts = (lo + rng.random((n, 3)) * (hi - lo)).astype(np.float32)
    pts[::4] = g.position[rng.integers(0, g.position.shape[0], pts[::4].shape[0])] * np.float32(1.01) + np.float32(0.01)
    if n > 30:
        pts[3:6] = [[np.nan, 0, 0], [0, np.inf, 0], [3e38, 0, 0]]
    d = torch.from_numpy(pts).to(cuda)
    for far in (math.inf, 1.5, 0.0):
        bvh.set_traversal(closest=0)
        want = bvh.closest_point_batch(d, 1e-30, far).view(torch.int32)
        for kw in (dict(closest=0), dict(closest=1), dict(closest=1, tile=32, tile_rows=4), dict(closest=2)):
            bvh.set_traversal(**kw)
            got = bvh.closest_point_batch(d, 0.0, far)
            bvh.synchronize()
            assert torch.equal(got.view(torch.int32), want), (far, kw)


@pytest.mark.parametrize("mesh", ["triangle", "leaf40", "leaves40", "groups", "plain"])
@pytest.mark.parametrize("n", [1, 5, 33, 32768, 32769, 65537])
def test_shapes_match(pkg, orc, cuda, mesh, n):
    """Any-hit spheres and oriented boxes, the whole warp and four lanes per shape: spheres as the
    per-sphere child-pair walk counts them, boxes as the oracle answers, with boxes that rest on the
    mesh's vertices (undecided in float32) among them."""
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    ref = orc.OracleBVH.from_serialized(bvh._roots, g.index, bvh._indirectBuffer, g.position)
    rng = np.random.default_rng(n)
    lo, hi = g.position.min(0) - 1, g.position.max(0) + 1
    c = (lo + rng.random((n, 3)) * (hi - lo)).astype(np.float32)
    corner = g.position[g.index[rng.integers(0, len(g.index), n)]]
    spheres = np.concatenate([c, np.exp(rng.uniform(-4, 1, (n, 1)))], 1).astype(np.float32)
    spheres[::9, 3] = 0.0
    spheres[::9, :3] = corner[::9]
    half = (rng.random((n, 3)) * 0.9 + 0.05).astype(np.float32)
    boxes = np.zeros((n, 24), np.float32)
    boxes[:, 0:3], boxes[:, 4:7] = -half, half
    boxes[:, 8] = boxes[:, 13] = boxes[:, 18] = boxes[:, 23] = 1.0
    a = rng.uniform(0, 6, n)
    boxes[::2, 8], boxes[::2, 9], boxes[::2, 12], boxes[::2, 13] = (v[::2] for v in (
        np.cos(a), np.sin(a), -np.sin(a), np.cos(a)))
    boxes[:, 20:23] = c
    rest = np.arange(n) % 3 == 1          # one face through a vertex of the mesh, exactly or nearly
    boxes[rest, 20:23] = corner[rest]
    boxes[rest, 20] += half[rest, 0] * np.float32(1 + 1e-7)
    boxes[::11, 19] = 0.01                # projective
    want_s, want_b = bvh.sphere_triangles_batch(spheres, cap=1)[0] > 0, ref.intersects_box(boxes)
    got_s = bvh.intersects_sphere_batch(torch.from_numpy(spheres).to(cuda)).cpu().numpy().astype(bool)
    got_b = bvh.intersects_box_batch(torch.from_numpy(boxes).to(cuda)).cpu().numpy().astype(bool)
    bvh.synchronize()
    assert np.array_equal(got_s, want_s)
    assert np.array_equal(got_b, want_b)


@pytest.mark.parametrize("n", [100, 30_000, 140_000])
def test_boxes_outside_their_parents(pkg, cuda, n):
    """A tree from a file whose inner boxes do not hold their children's: rays miss what the
    child-pair kernel misses."""
    import torch

    g, _ = _mesh(pkg, "plain")
    data = pkg.MeshBVH.serialize(pkg.MeshBVH(g, {"strategy": pkg.SAH}))
    nodes = np.frombuffer(data["roots"][0], np.float32).reshape(-1, 8).copy()
    count = nodes.view(np.uint32)[:, 7]
    for k in range(1, 40):
        if count[k] >> 16 != 0xFFFF:          # an inner node
            nodes[k, 3:6] = 0.5 * (nodes[k, 0:3] + nodes[k, 3:6])
    data["roots"] = [nodes.tobytes()]
    bvh = pkg.MeshBVH.deserialize(data, g)
    rays = torch.from_numpy(_rays(pkg, n)).to(cuda)
    bvh.set_traversal(0, 1)
    want = bvh.raycast_first_batch(rays)
    bvh.set_traversal(1, 1)
    got = bvh.raycast_first_batch(rays)
    bvh.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    full = pkg.MeshBVH(g, {"strategy": pkg.SAH}).raycast_first_batch(rays)
    assert not torch.equal(full.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("n", [32, 1000, 5000, 131072, 200_001])
@pytest.mark.parametrize("near,far", [(0.0, math.inf), (30.0, 900.0)])
def test_instances_match_fewer_rays_per_call(pkg, cuda, n, near, far):
    """Instanced raycastFirst, phased: the records of calls of fewer than 32 rays, which go one thread per ray."""
    import torch

    batched = importlib.import_module(pkg.__name__ + ".batched")
    rng = np.random.default_rng(n)
    batch = batched.BatchedMeshBVH([_mesh(pkg, k)[0] for k in ("plain", "leaf40", "triangle")], {"strategy": pkg.SAH})
    batch.set_leaf_size(3 if n % 2 else 0)
    k = 70
    q, _ = np.linalg.qr(rng.standard_normal((k, 3, 3)))
    m = np.zeros((k, 16))
    for c in range(3):
        m[:, 4 * c:4 * c + 3] = q[:, :, c] * rng.uniform(0.4, 2.0, (k, 1))
    m[:, 12:15] = rng.uniform(-60, 60, (k, 3))
    m[:, 15] = 1
    m[1], geometry = m[0], rng.integers(0, 3, k).astype(np.uint32)
    geometry[1] = geometry[0]              # two instances in one place: the lower index
    scene = batch.instances(geometry, m)
    o = rng.standard_normal((n, 3))
    o *= 150 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(-60, 60, (n, 3)) - o
    d[::2] /= np.linalg.norm(d[::2], axis=1, keepdims=True)
    rays = torch.from_numpy(np.concatenate([o, d], 1).astype(np.float32)).to(cuda)
    hits, inst = scene.raycast_first(rays, 2, near, far)
    torch.cuda.synchronize()
    assert (inst != -1).any()
    step = max(1, n // 300)
    for i in range(0, n, 31 * step):
        one = rays[i:i + 31].clone()
        h, k1 = scene.raycast_first(one, 2, near, far)
        torch.cuda.synchronize()
        assert torch.equal(k1, inst[i:i + 31])
        assert torch.equal(h.view(torch.int32), hits[i:i + 31].view(torch.int32))


@pytest.mark.parametrize("n", [1, 511, 512, 513])
@pytest.mark.parametrize("config", [(0, 1), (1, 1), (1, 1, 16, 0, 1)])
def test_host_rays_match_device_rays(pkg, cuda, n, config):
    """Up to 512 host rays are read and written in page-locked memory, more through device buffers."""
    import torch

    bvh = pkg.MeshBVH(_mesh(pkg, "plain")[0], {"strategy": pkg.SAH})
    bvh.set_traversal(*config)
    rays = _rays(pkg, n)
    want = bvh.raycast_first_batch(torch.from_numpy(rays).to(cuda))
    bvh.synchronize()
    for _ in range(2):
        got = np.ascontiguousarray(bvh.raycast_first_batch(rays)).view(np.int32).reshape(n, 8)
        assert np.array_equal(got, want.view(torch.int32).cpu().numpy())
